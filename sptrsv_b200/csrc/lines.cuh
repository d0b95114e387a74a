// lines.cuh — drop-in solves (ORDER, MULTIROW) of stencils, straight from the
// caller's CSR: grid lines instead of levels.
//
// The analysis (k_line_check) has found that lines of w rows cut the matrix so
// that a row reads, besides the row before it in its line, only rows before its
// chunk of 32.  CTA g takes the lines G g ... G g + G - 1, one warp a line,
// their x in shared memory; a warp goes along its line chunk by chunk, a lane a
// row, and closes a chunk by an affine scan over x_j = a_j + beta_j x_j-1 (as
// k_sptrsv_wave4, whose comment says why the order of loads and stores is held
// by __syncwarp()).  Every column lies in an earlier line or an earlier chunk of
// the same line, groups are taken in order and the CTAs are co-resident, so the
// lowest unfinished chunk never waits on an unfinished one.
//
// The entries of a chunk's rows are contiguous in the CSR: they and b are copied
// to shared memory two chunks ahead by cp.async, their row pointers loaded
// three ahead.
//
// Bound: the chain of lines.  A level of a 2048 x 2048 grid costs the level
// order 0.91 us (a hop through L2 and the row behind it), 4095 levels; a line
// here 0.4 us (most of them a hop in shared memory), 2048 lines.  FP64, MULTIROW
// before and after: 2048 x 2048 3756 -> 903 us, 1000 x 900 1671 -> 376 us, 333 x
// 277 503 -> 126 us, 101 x 90 x 97 334 -> 145 us, 128^3 480 -> 198 us.
#pragma once

#include "solve_kernels.cuh"

namespace sptrsv {

constexpr int kLineG = 8;  // most lines of a CTA

// Entries of 32 rows of up to U off-diagonals, b behind them; two of these a warp.
constexpr __host__ __device__ size_t line_stage_bytes(int U)
{
    return (size_t)32 * ((U + 1) * (sizeof(double) + sizeof(int)) + sizeof(double));
}

template <int U>
__global__ void __launch_bounds__(32 * kLineG, 1)
    k_sptrsv_lines(const int* __restrict__ rowptr, const int* __restrict__ col, const double* __restrict__ val, int n, int w,
                   int G, const double* __restrict__ b, double* x, DevStatus* st, unsigned long long budget)
{
    constexpr int EC = 32 * (U + 1);  // entries of a stage
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int abort_flag;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    volatile double* xs = reinterpret_cast<double*>(smem_raw);
    double* sval = reinterpret_cast<double*>(smem_raw) + (size_t)G * w + (size_t)wib * (2 * line_stage_bytes(U) / 8);
    double* sb = sval + 2 * EC;
    int* scol = reinterpret_cast<int*>(sb + 2 * 32);
    if (threadIdx.x == 0) abort_flag = 0;
    const int per = G * w, ngroups = (n + per - 1) / per;
    bool failed = false;
    for (int g = blockIdx.x; g < ngroups; g += gridDim.x) {
        const int R0 = g * per, rows = min(per, n - R0);
        for (int t = threadIdx.x; t < rows; t += blockDim.x) xs[t] = sentinel_value<double>();
        __syncthreads();
        const int line0 = R0 + wib * w, lend = min(line0 + w, n);
        if (wib * w < rows) {
            // this lane's row of the chunk at c0: its entries [s, e), none past the line's end
            auto ptrs = [&](int c0, int& s, int& e) {
                s = e = 0;
                if (c0 + lane < lend) {
                    asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(s) : "l"(rowptr + c0 + lane) : "memory");
                    asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(e) : "l"(rowptr + c0 + lane + 1) : "memory");
                }
            };
            auto stage = [&](int k, int c0, int s, int e) {
                if (c0 < lend) {
                    const int base = __shfl_sync(FULL, s, 0), cnt = __reduce_max_sync(FULL, e) - base;
#pragma unroll
                    for (int j = 0; j <= U; j++)
                        if (j * 32 + lane < cnt) {
                            cp_async_ca(scol + k * EC + j * 32 + lane, col + base + j * 32 + lane);
                            cp_async_ca(sval + k * EC + j * 32 + lane, val + base + j * 32 + lane);
                        }
                    if (c0 + lane < lend) cp_async_ca(sb + k * 32 + lane, b + c0 + lane);
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            int s, e, s1, e1, s2, e2;
            ptrs(line0, s, e);
            ptrs(line0 + 32, s1, e1);
            stage(0, line0, s, e);
            stage(1, line0 + 32, s1, e1);
            ptrs(line0 + 64, s2, e2);
            double carry = 0;
            for (int c0 = line0, buf = 0; c0 < lend; c0 += 32, buf ^= 1) {
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                __syncwarp();
                const int r = c0 + lane;
                const bool act = r < lend;
                const int base = __shfl_sync(FULL, s, 0), off = buf * EC - base;
                double a = 0, inv = 0, lsub = 0, v[U], xv[U];
                int c[U];
                const int cnt = e - s - 1;
                // the form that the analysis found, or the CSR has changed since
                bool sub = false, glob = false, bad = act && (cnt < 0 || cnt > U || s < base || e - base > EC);
                if (act && !bad) {
                    a = sb[buf * 32 + lane];
                    inv = 1.0 / sval[off + s + cnt];
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    c[u] = -1;
                    v[u] = 0;
                    xv[u] = 0;
                    if (u < cnt && !bad) {
                        c[u] = scol[off + s + u];
                        v[u] = sval[off + s + u];
                        if (c[u] == r - 1 && r > line0) {
                            lsub = v[u];
                            sub = true;
                            c[u] = -1;
                        }
                        glob |= c[u] >= 0 && c[u] < R0;
                    }
                }
#pragma unroll
                for (int u = 0; u < U; u++) bad |= c[u] >= c0;
                if (__any_sync(FULL, bad)) {
                    if (bad) report(st, SPTRSV_ERR_INVALID_CSR, r);
                    failed = true;
                    break;
                }
                glob = __any_sync(FULL, glob);
                unsigned it = 0;
                unsigned long long t0 = 0;
                if (glob) {
#pragma unroll
                    for (int u = 0; u < U; u++)
                        if (c[u] >= 0 && c[u] < R0) xv[u] = ld_relaxed(x + c[u]);
                }
                // what does not depend on x
                const double beta = sub ? -lsub * inv : 0.0;
                const bool steep = __any_sync(FULL, !(fabs(beta) <= 1.0));
                double M[5], B = beta;
#pragma unroll
                for (int d = 0; d < 5; d++) {
                    M[d] = B;
                    const double up = __shfl_up_sync(FULL, B, 1 << d);
                    if (lane >= (1 << d)) B *= up;
                }
                if (glob) {
                    while (true) {
                        bool pend = false;
#pragma unroll
                        for (int u = 0; u < U; u++) pend |= is_pending(xv[u]);
                        if (!__any_sync(FULL, pend)) break;
                        if ((++it & 63u) == 0 && give_up(t0, st, budget, c0)) {
                            failed = true;
                            break;
                        }
#pragma unroll
                        for (int u = 0; u < U; u++)
                            if (c[u] >= 0 && c[u] < R0) xv[u] = ld_relaxed(x + c[u]);
                    }
                }
                while (!failed) {
                    bool pend = false;
#pragma unroll
                    for (int u = 0; u < U; u++)
                        if (c[u] >= R0) xv[u] = xs[c[u] - R0];
#pragma unroll
                    for (int u = 0; u < U; u++) pend |= is_pending(xv[u]);
                    if (!__any_sync(FULL, pend)) break;
                    if ((++it & 63u) == 0 && give_up(t0, st, budget, c0)) failed = true;
                }
                if (failed) break;
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (c[u] >= 0) a -= v[u] * xv[u];
                double A = a * inv;
                if (lane == 0) A += beta * carry;
#pragma unroll
                for (int d = 0; d < 5; d++) {
                    const double up = __shfl_up_sync(FULL, A, 1 << d);
                    if (lane >= (1 << d)) A += M[d] * up;
                }
                // factors above 1 are not multiplied up, and an infinity times a product that
                // underflowed would be NaN: such a chunk goes row by row
                if (__any_sync(FULL, !finite_bits(A)) || steep) {
                    double t = carry;
                    for (int l = 0; l < 32; l++) {
                        t = (sub ? a - lsub * t : a) * inv;
                        if (lane == l) A = publishable(t);
                        t = __shfl_sync(FULL, t, l);
                    }
                }
                if (act) xs[r - R0] = A;
                __syncwarp();
                if (act) st_relaxed(x + r, A);
                carry = __shfl_sync(FULL, A, 31);
                __syncwarp();
                stage(buf, c0 + 64, s2, e2);
                s = s1, e = e1, s1 = s2, e1 = e2;
                ptrs(c0 + 96, s2, e2);
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
        if (failed && lane == 0) abort_flag = 1;
        __syncthreads();
        if (abort_flag) return;
    }
}

}  // namespace sptrsv
