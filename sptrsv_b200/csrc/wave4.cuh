// wave4.cuh — the WAVE schedule's kernel for block systems of 2D stencils with
// one coupling outside the line (five points).
//
// Groups of grid lines, one CTA a group, one warp a line, the group's x in
// shared memory (see strip.cu).  A line is cut into chunks of 128 consecutive
// rows, lane j owning the rows 4 j .. 4 j + 3.  Inside a chunk a row depends on
// the row before it only (the chunk's first row on the chunk before), so a
// chunk is the first-order recurrence x_j = a_j + beta_j x_j-1: each lane
// composes its four rows in sequence, five steps of an affine scan over the
// lanes give every lane the row before its first, and its rows follow.
// Everything of the scan that does not depend on x (products of beta over 2^d
// lanes, and over a lane's rows) is computed before the chunk waits for the
// line above.  A chunk's arrays are prefetched to L2 two chunks ahead and loaded
// into one set of registers once the chunk before has stored its x (loads that
// rotate through two sets are waited for at every copy).
//
// With many blocks the solve is bound by what a chunk costs its SM and by the
// lag from a line's chunk to the next line's (about 0.35 us in a CTA), not by
// one chain, so a chunk of 128 rows beats the one-row-a-lane form, which spends
// the same scan on 32.  FP64 / refined solve, us, one row a lane -> here, 4
// lines a CTA (with the gather and scatter of the block system, which this
// kernel does not need):
//   2048 x 2048, 16 blocks  237 / 812 -> 128 / 530,  32 blocks  241 / 754 -> 100 / 465
//   1000 x 900,  16 blocks  106 / 350 ->  67 / 216
//   333 x 277,   16 blocks   53 / 156 ->  41 / 116
// An unpartitioned system is one chain of hops from group to group, where a hop
// costs this kernel more (2048 x 2048, 4 lines a CTA: 856 against 997 us;
// 101 x 90 x 97, two couplings: 144 against 225 us): it keeps the other form.
//
// What keeps the lag short is the order of instructions: a chunk's x is stored
// before anything of the next chunk is loaded, held there by __syncwarp() (left
// to the compiler, loads and address arithmetic moved ahead of the store: 0.62
// instead of 0.42 us a line), and the next chunk's row range is loaded a chunk
// earlier, as waiting for it would hold up the loads that need it.
//
// Slots: chunk q's row p (lane p / 4, i = p % 4) is slot 128 q + p, with
// inv = 1 / L_rr, lsub = L_r,r-1 (0 for a line's first row) and the one entry
// outside the line, ev and ecol.  A column inside the row's group is ~place in
// shared memory, another its place in xp; an unused entry has value 0 and the
// place of a constant 0.  A chunk's places are transposed (row p at base +
// i * lanes + lane), so that a line reads the line above without bank conflicts.
//
// xp is the chunks that another group reads (all-ones until known), packed.
// Group g's rows are the outer plan's rows gmap[2 g] ...: b is read and the
// results are written there directly, from the group's row gmap[2 g + 1] on (the
// ones before are warm-up rows).
#pragma once

#include <string.h>

#include "plan.h"
#include "solve_kernels.cuh"

namespace sptrsv {

constexpr int kWave4Q = 4;              // rows a lane
constexpr int kWave4C = 32 * kWave4Q;   // rows a chunk

template <typename V>
struct Wave4Mat {
    const V* __restrict__ inv;
    const V* __restrict__ lsub;
    const V* __restrict__ ev;
    const int* __restrict__ ecol;
    const int4* __restrict__ chunk;  // first row, rows, first place, place in xp (-1: no other group reads it)
    const int* __restrict__ runc;    // first chunk of each run
    const int* __restrict__ grun;    // first run of each group
    const int* __restrict__ grow;    // first row of each group
    const int* __restrict__ gseq;    // processing order of the groups (null: natural)
    const int* __restrict__ gmap;    // per group: outer row of its first row, its first real row
    int zero;                        // the place of the constant 0
};

// Read-only loads that stay where they are written: moved up by the compiler,
// ahead of a chunk's own x, they cost the line below half as much again.
template <typename E, int N>
__device__ __forceinline__ void ldg_vec(const E* p, E (&r)[N])
{
    static_assert(sizeof(E) * N % 16 == 0 || sizeof(E) * N == 8 || N == 1, "whole vectors");
    if constexpr (sizeof(E) * N == 4) {
        unsigned v;
        asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
        memcpy(&r[0], &v, 4);
    } else if constexpr (sizeof(E) * N == 8) {
        uint2 v;
        asm volatile("ld.global.nc.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
        memcpy(&r[0], &v, 8);
    } else {
#pragma unroll
        for (int k = 0; k < (int)(sizeof(E) * N / 16); k++) {
            uint4 v;
            asm volatile("ld.global.nc.v4.b32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                         : "l"(reinterpret_cast<const uint4*>(p) + k)
                         : "memory");
            memcpy(&r[k * (16 / sizeof(E))], &v, 16);
        }
    }
}

__device__ __forceinline__ void st_relaxed2(double* p, double a, double b)
{
    asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(a), "d"(b) : "memory");
}
__device__ __forceinline__ void st_relaxed2(float* p, float a, float b)
{
    asm volatile("st.relaxed.gpu.global.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(a), "f"(b) : "memory");
}

template <typename V, typename T>
struct Wave4Op {
    static constexpr int Q = kWave4Q;
    V inv[Q], lsub[Q], ev[Q];
    int ec[Q];
    T b[Q];
    double x64[Q];  // OUT_ADD64
    int4 m;
};

template <typename V, typename T, typename BT, int OUT, bool STREAM>
__global__ void __launch_bounds__(512, 1) k_sptrsv_wave4(Wave4Mat<V> w, int ngroups, const BT* __restrict__ b, T* xp,
                                                        T* xo, double* x64, DevStatus* st, unsigned long long budget,
                                                        const int* bflag, int seg_rows, int epoch, double* hx)
{
    constexpr int Q = kWave4Q, C = kWave4C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int abort_flag;
    const unsigned FULL = 0xffffffffu;
    volatile T* xs = reinterpret_cast<volatile T*>(smem_raw);
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        xs[w.zero] = (T)0;
    }
    int seg_ok = -1;  // streamed b: the last segment whose flag this lane saw set
    bool failed = false;
    for (int k = blockIdx.x; k < ngroups; k += gridDim.x) {
        const int g = w.gseq ? __ldg(w.gseq + k) : k;
        const int run0 = __ldg(w.grun + g), run1 = __ldg(w.grun + g + 1);
        const int r0 = __ldg(w.grow + g);
        const int shift = __ldg(w.gmap + 2 * g) - r0;         // row -> row of b and of the results
        const int real = r0 + __ldg(w.gmap + 2 * g + 1);      // first row with results
        const int4 last = __ldg(w.chunk + __ldg(w.runc + run1) - 1);
        const int places = last.z + (last.y + Q - 1) / Q * Q;
        for (int t = threadIdx.x; t < places; t += blockDim.x) xs[t] = sentinel_value<T>();
        __syncthreads();
        const int run = run0 + wib;
        if (run < run1) {
            const int q0 = __ldg(w.runc + run), q1 = __ldg(w.runc + run + 1);
            T carry = (T)0;
            int4 mn = __ldg(w.chunk + q0);  // of the chunk that load() takes next: never waited for there
            auto load = [&](Wave4Op<V, T>& z, int q) {
                z.m = mn;
                if (q + 1 < q1) mn = __ldg(w.chunk + q + 1);
                const size_t s = (size_t)q * C + lane * Q;
                ldg_vec(w.inv + s, z.inv);
                ldg_vec(w.lsub + s, z.lsub);
                ldg_vec(w.ev + s, z.ev);
                ldg_vec(w.ecol + s, z.ec);
                const int rows = min(Q, z.m.y - lane * Q);  // of this lane (may be <= 0)
                const int rb = z.m.x + lane * Q + shift;
                if (STREAM && bflag) {
                    const int sg = rows > 0 ? (rb + rows - 1) / seg_rows : seg_ok;  // segments arrive in order
                    const bool need = sg != seg_ok;
                    if (__any_sync(FULL, need)) {
                        if (!warp_wait_flag(need, bflag + (need ? sg : 0), epoch, st, budget, rb)) failed = true;
                        if (need) seg_ok = sg;
                    }
                }
#pragma unroll
                for (int i = 0; i < Q; i++) z.b[i] = (T)0;
                if (OUT == OUT_ADD64) {
#pragma unroll
                    for (int i = 0; i < Q; i++)
                        if (i < rows && rb - shift + i >= real) z.x64[i] = x64[rb + i];
                }
                if (!STREAM && rows == Q && ((uintptr_t)(b + rb) & 15) == 0) {
                    BT v[Q];
                    ldg_vec(b + rb, v);
#pragma unroll
                    for (int i = 0; i < Q; i++) z.b[i] = (T)v[i];
                } else {
#pragma unroll
                    for (int i = 0; i < Q; i++)
                        if (i < rows) {
                            BT v[1];
                            if (STREAM) v[0] = ld_relaxed(b + rb + i);
                            else ldg_vec(b + rb + i, v);
                            z.b[i] = (T)v[0];
                        }
                }
            };
            auto ahead = [&](int q) {  // chunk q to L2: a lane touches a 128-byte line
                const size_t s = (size_t)q * C;
                constexpr int LV = C * sizeof(V) / 128;  // lines of each of inv, lsub, ev
                static_assert(3 * LV + C / 32 <= 32, "a lane a line");
                const void* p = w.ecol + s + (lane - 3 * LV) * 32;
                if (lane < 3 * LV) p = (lane < LV ? w.inv : lane < 2 * LV ? w.lsub : w.ev) + s + lane % LV * (128 / sizeof(V));
                if (lane < 3 * LV + C / 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
                if (!STREAM) {
                    const int rb = __ldg(&w.chunk[q].x) + shift, rows = __ldg(&w.chunk[q].y);
                    const int t = lane * (128 / (int)sizeof(BT));
                    if (t < rows) asm volatile("prefetch.global.L2 [%0];" ::"l"(b + rb + t));
                }
            };
            Wave4Op<V, T> z;
            if (q0 + 1 < q1) ahead(q0 + 1);
            load(z, q0);
            for (int q = q0; q < q1 && !failed; q++) {
                if (q + 2 < q1) ahead(q + 2);
                // x of other groups, long known except on a group's first line: under way first
                bool glob = false;
#pragma unroll
                for (int i = 0; i < Q; i++) glob |= z.ec[i] >= 0;
                glob = __any_sync(FULL, glob);
                T xv[Q];
                if (glob) {
#pragma unroll
                    for (int i = 0; i < Q; i++) {
                            xv[i] = (T)0;
                            if (z.ec[i] >= 0) xv[i] = ld_relaxed(xp + z.ec[i]);
                        }
                }
                // what does not depend on x
                T P[Q], M[5];
                P[0] = -(T)z.lsub[0] * (T)z.inv[0];
                T be[Q];
                be[0] = P[0];
#pragma unroll
                for (int i = 1; i < Q; i++) {
                    be[i] = -(T)z.lsub[i] * (T)z.inv[i];
                    P[i] = P[i - 1] * be[i];
                }
                T Bd = P[Q - 1];
#pragma unroll
                for (int d = 0; d < 5; d++) {
                    M[d] = Bd;
                    const T up = __shfl_up_sync(FULL, Bd, 1 << d);
                    if (lane >= (1 << d)) Bd *= up;
                }
                unsigned it = 0;
                unsigned long long t0 = 0;
                if (!glob) {
                    while (true) {
                        bool pend = false;
#pragma unroll
                        for (int i = 0; i < Q; i++) xv[i] = xs[~z.ec[i]];
#pragma unroll
                        for (int i = 0; i < Q; i++) pend |= is_pending(xv[i]);
                        if (!__any_sync(FULL, pend)) break;
                        if ((++it & 63u) == 0 && give_up(t0, st, budget, z.m.x)) {
                            failed = true;
                            break;
                        }
                    }
                } else {
                    while (true) {
                        bool pend = false;
#pragma unroll
                        for (int i = 0; i < Q; i++) pend |= is_pending(xv[i]);
                        if (!__any_sync(FULL, pend)) break;
                        if ((++it & 63u) == 0 && give_up(t0, st, budget, z.m.x)) {
                            failed = true;
                            break;
                        }
#pragma unroll
                        for (int i = 0; i < Q; i++)
                                if (z.ec[i] >= 0) xv[i] = ld_relaxed(xp + z.ec[i]);
                    }
                    while (!failed) {
                        bool pend = false;
#pragma unroll
                        for (int i = 0; i < Q; i++)
                                if (z.ec[i] < 0) xv[i] = xs[~z.ec[i]];
#pragma unroll
                        for (int i = 0; i < Q; i++) pend |= is_pending(xv[i]);
                        if (!__any_sync(FULL, pend)) break;
                        if ((++it & 63u) == 0 && give_up(t0, st, budget, z.m.x)) failed = true;
                    }
                }
                if (failed) break;
                T a[Q];
#pragma unroll
                for (int i = 0; i < Q; i++) {
                    a[i] = (z.b[i] - (T)z.ev[i] * xv[i]) * (T)z.inv[i];
                }
                const int4 m = z.m;
                double sum[Q];
                if (OUT == OUT_ADD64) {
#pragma unroll
                    for (int i = 0; i < Q; i++) sum[i] = z.x64[i];
                }
                T c[Q];
                c[0] = a[0];
#pragma unroll
                for (int i = 1; i < Q; i++) c[i] = a[i] + be[i] * c[i - 1];
                T A = c[Q - 1];
                if (lane == 0) A += P[Q - 1] * carry;
#pragma unroll
                for (int d = 0; d < 5; d++) {
                    const T up = __shfl_up_sync(FULL, A, 1 << d);
                    if (lane >= (1 << d)) A += M[d] * up;
                }
                T in = __shfl_up_sync(FULL, A, 1);
                if (lane == 0) in = carry;
                // An infinity times a product that underflowed would be NaN: a chunk with a row that
                // is not finite goes row by row (any such row shows in its lane's last).
                const bool odd = __any_sync(FULL, !finite_bits(A));
                T v[Q];
#pragma unroll
                for (int i = 0; i < Q; i++) v[i] = c[i] + P[i] * in;
                if (odd) {
                    A = carry;
                    for (int l = 0; l < 32; l++) {
#pragma unroll
                        for (int i = 0; i < Q; i++) {
                            A = a[i] + be[i] * A;
                            if (lane == l) v[i] = publishable(A);
                        }
                        A = __shfl_sync(FULL, A, l);
                    }
                }
                const int rows = min(Q, m.y - lane * Q), lanes = (m.y + Q - 1) / Q;
                const int r = m.x + lane * Q;
#pragma unroll
                for (int i = 0; i < Q; i++)
                    if (i < rows) xs[m.z + i * lanes + lane] = v[i];
                __syncwarp();  // and nothing of what follows before it
                carry = __shfl_sync(FULL, A, 31);
                auto store = [&](T* p) {
                    if (Q > 1 && rows == Q && ((uintptr_t)p & (2 * sizeof(T) - 1)) == 0) {
#pragma unroll
                        for (int i = 0; i + 1 < Q; i += 2) st_relaxed2(p + i, v[i], v[i + 1]);
                    } else {
#pragma unroll
                        for (int i = 0; i < Q; i++)
                            if (i < rows) st_relaxed(p + i, v[i]);
                    }
                };
                if (m.w >= 0) store(xp + m.w + lane * Q);
                // the next chunk's operands, in L2 by now: after the stores that others wait for
                __syncwarp();
                if (!STREAM && q + 1 < q1) load(z, q + 1);
                if (OUT == OUT_X && !(STREAM && hx)) {
                    if (r >= real) store(xo + r + shift);
                    else {
#pragma unroll
                        for (int i = 0; i < Q; i++)
                            if (i < rows && r + i >= real) xo[r + shift + i] = v[i];
                    }
                }
                if (OUT != OUT_X) {
#pragma unroll
                    for (int i = 0; i < Q; i++)
                        if (i < rows && r + i >= real) {
                            if (OUT == OUT_SET64) x64[r + shift + i] = (double)v[i];
                            else x64[r + shift + i] = sum[i] + (double)v[i];
                        }
                }
                if (STREAM && q + 1 < q1) load(z, q + 1);  // may wait for b to arrive
            }
        }
        if (failed && lane == 0) abort_flag = 1;
        __syncthreads();
        if (abort_flag) return;
        if (STREAM && hx) {
            // the group's results to the caller's array in one go: chunk by chunk, rows in order
            const int c0 = __ldg(w.runc + run0), c1 = __ldg(w.runc + run1);
            for (int q = c0 + wib; q < c1; q += blockDim.x >> 5) {
                const int4 m = __ldg(w.chunk + q);
                const int lanes = (m.y + Q - 1) / Q;
                for (int t = lane; t < m.y; t += 32)
                    if (m.x + t >= real) hx[m.x + t + shift] = (double)xs[m.z + (t % Q) * lanes + t / Q];
            }
            __syncthreads();
        }
    }
}

}  // namespace sptrsv
