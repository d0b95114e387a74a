// analysis.cu — GPU analysis pass, bit-exact with the reference's
// multirow_analysis_base_GPU (analysis/analysis_csr.cu:272-410).
//
// Steps (reference line in brackets):
//  0. CSR validation: lower triangular, sorted columns, diagonal last.  The
//     reference trusts its input and hangs on a bad one; here a bad matrix
//     is an error return.
//  1. Levels [:104-185]: level[i] = 1 + max(level[j]) over the off-diagonal
//     columns j of row i.  This is a max-plus triangular solve, done with the
//     same sync-free pattern as the numeric solve: a persistent grid walks the
//     rows in natural order (a topological order), each row polls its
//     dependencies' levels (0 = not yet written) with bounded relaxed loads.
//     nlevs = max level [:305] via one atomicMax per warp.
//  2. Key = 7*(level-1) + bucket(offdiag count) [:12-32, :53-57, :307-332]
//     and per-key row counts (the reference's sort + reduce_by_key + scatter,
//     :336-348) with warp-aggregated atomics.
//  3. iorder = rows stably sorted by key [:350-352]: the stable LSD radix
//     sort of util.cu on (key, row).
//  4. Multirow warp map [:354-385, kernel_base :244-270]: warps per key =
//     ceil(count * lanes / 32), two exclusive scans, then one thread per warp
//     writes ibase_row / ivect_size_warp.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <initializer_list>
#include <vector>

#include "blocks.h"
#include "internal.h"

namespace sptrsv {

namespace {

// bucket of a row by its off-diagonal count (vect_size_calculator, :12-32)
__device__ __forceinline__ int bucket_of(int nnz_off)
{
    if (nnz_off == 0) return 6;
    if (nnz_off == 1) return 0;
    if (nnz_off <= 2) return 1;
    if (nnz_off <= 4) return 2;
    if (nnz_off <= 8) return 3;
    if (nnz_off <= 16) return 4;
    return 5;
}

// res[0] = error flag, res[1] = first bad row (starts at INT_MAX)
__global__ void k_validate(const int* __restrict__ rowptr, const int* __restrict__ col, int n, int nnz, int* res)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int s = rowptr[i], e = rowptr[i + 1];
        bool bad = (i == 0 && s != 0) || e <= s || e > nnz || s < 0;
        if (!bad) {
            bad = col[e - 1] != i;
            int prev = -1;
            for (int p = s; p < e - 1 && !bad; p++) {
                int c = col[p];
                if (c <= prev || c >= i) bad = true;
                prev = c;
            }
        }
        if (bad) {
            atomicOr(res, 1);
            atomicMin(res + 1, i);
        }
    }
}

// Persistent sync-free level computation over natural-order groups, one
// thread per row.  CTA g takes the groups g, g + G, ...: kLvGroup consecutive
// rows (or, with a task table, the rows [task_r0[t], task_r0[t] +
// task_cnt[t]); any order in which every row's dependencies lie in earlier
// tasks or earlier in its own is deadlock-free).  The group's levels live in
// shared memory (0 = not yet known), so a dependency inside the group is a
// shared-memory poll; others are polled in global memory.
//
// Every lane walks its own row and publishes as soon as the row is done: a
// warp that holds the end of one grid line and the start of the next must
// not make the second wait for the first (solving a warp's rows in order did,
// and strung all lines of a grid behind one another: 322 ms on a 1023 x 1025
// grid).  Columns inside the row's own warp are not polled.  Where they are
// the row before only (stencils), a max-plus prefix scan over the lanes closes
// the warp, the level of the row before the warp entering last, so a grid
// line costs one hop per warp and not 32 dependent steps.  Otherwise one pass
// over the lanes that are read, in order, hands each finished level to the
// lanes that read it (about 45 cycles a lane read, against 600 for a poll
// round through shared memory), once all rows' outside columns are known or
// when some are long in coming.
//
// Before it looks at all its columns a warp waits for one word: the smallest,
// over its rows without a column inside the warp, of the row's largest
// column.  The warp's first finished row is one of those, and thousands of
// warps that wait far from the front then cost one L2 sector a poll each.
//
// Bound: hops.  A value written by one SM is seen by another 707 cycles later
// (measured, B200), a line costs about 1,700.  Kernel times before and after:
// 1023 x 1025 grid with holes 322 -> 2.0 ms, 2048 x 2048 grid 2.7 -> 1.9 ms,
// 101 x 90 x 97 grid 431 -> 0.26 ms, banded n = 1e5 (8 in 256) 44.7 -> 4.0 ms,
// banded n = 3e5 (4-8 in 16) 132 -> 15.7 ms, Zipf n = 2e6 42 -> 1.5 ms, dense
// 32-row blocks n = 5e5 58 -> 48 us.
constexpr int kLvStall = 16;  // polls without an answer after which a warp looks for rows that can do without

template <int U>
__global__ void __launch_bounds__(kLvGroup) k_levels(const int* __restrict__ rowptr, const int* __restrict__ col,
                                                     int n, int* level, int* nlevs, DevStatus* st,
                                                     unsigned long long budget, const int* __restrict__ task_r0,
                                                     const int* __restrict__ task_cnt, long long ntasks)
{
    __shared__ volatile int lv[kLvGroup];
    __shared__ int abort_flag;
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
    const unsigned upto = FULL >> (31 - lane);  // lanes 0..lane
    int my_max = 0;
    if (tid == 0) abort_flag = 0;
    for (long long t = blockIdx.x; t < ntasks; t += gridDim.x) {
        const int R0 = task_r0 ? __ldg(task_r0 + t) : (int)(t * kLvGroup);
        const int cnt = task_r0 ? __ldg(task_cnt + t) : min(kLvGroup, n - R0);
        const int r = R0 + tid, w0 = R0 + wib * 32;
        const bool act = tid < cnt;
        lv[tid] = 0;
        int p = 0, e = 0;
        if (act) {
            p = __ldg(rowptr + r);
            e = __ldg(rowptr + r + 1) - 1;
        }
        int c[U], nb = 0, far = -1;
        unsigned pend = 0;    // columns of the batch outside the warp, not known yet
        unsigned inmask = 0;  // lanes of this warp the row reads and has not got yet
        auto batch = [&]() {
            nb = min(U, e - p);
            pend = 0;
#pragma unroll
            for (int u = 0; u < U; u++) {
                c[u] = -1;
                if (u < nb) {
                    c[u] = __ldg(col + p + u);
                    if (c[u] >= w0) inmask |= 1u << (c[u] - w0);
                    else pend |= 1u << u;
                }
            }
        };
        batch();
        const bool sub = lane > 0 && (inmask >> (lane - 1)) & 1u;
        // closed by the scan: no lane holds more than U columns, and none inside the warp but the row before
        const bool chain = __all_sync(FULL, e - p <= U && inmask == (sub ? 1u << (lane - 1) : 0u));
        unsigned cinbit = 0;  // chain: the column of lane 0 that is the row before the warp
#pragma unroll
        for (int u = 0; u < U; u++)
            if (pend >> u & 1u) {
                if (chain && lane == 0 && c[u] == w0 - 1) cinbit = 1u << u;
                else far = max(far, c[u]);
            }
        const bool cin = __shfl_sync(FULL, cinbit, 0) != 0;
        int word = __reduce_min_sync(FULL, act && inmask == 0 ? (cinbit ? w0 - 1 : far) : 0x7fffffff);
        if (cin && word == w0 - 1) {
            // the row before the warp comes last in a scan: the line above is awaited first
            const int above = __reduce_min_sync(FULL, far >= 0 ? far : 0x7fffffff);
            if (above != 0x7fffffff) word = above;
        }
        __syncthreads();  // lv is filled
        bool fail = false;
        unsigned it = 0, seen = 0;
        unsigned long long t0 = 0;
        if (word >= 0 && word != 0x7fffffff)
            while ((word >= R0 ? lv[word - R0] : ld_relaxed(level + word)) == 0)
                if ((++it & 63u) == 0 && give_up(t0, st, budget, w0)) {
                    fail = true;
                    break;
                }
        bool done = !act, ready = !act;  // ready: all columns outside the warp are known
        int m = 0, A = 0, vin = 0;
        // segments of rows linked to the row before: their first lanes, and this lane's
        const unsigned S = __ballot_sync(FULL, !sub) | 1u;
        const int start = 31 - __clz(S & upto);
        const unsigned need = upto & (FULL << start);
        bool all = true;  // poll every pending column
        bool stalled = false;
        while (!fail) {
            if (all) {
                int v[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    v[u] = 0;
                    if ((pend >> u & 1u) && c[u] < R0) v[u] = ld_relaxed(level + c[u]);
                }
#pragma unroll
                for (int u = 0; u < U; u++)
                    if ((pend >> u & 1u) && c[u] >= R0) v[u] = lv[c[u] - R0];
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (v[u] != 0) {
                        pend &= ~(1u << u);
                        if (cinbit >> u & 1u) vin = v[u];
                        else m = max(m, v[u]);
                    }
            }
            bool again = false;
            if (!ready && (pend & ~cinbit) == 0) {
                p += nb;
                if (p < e) {
                    batch();
                    again = true;
                } else {
                    ready = true;
                }
            }
            const unsigned R = __ballot_sync(FULL, ready);
            if (chain) {
                if (R != seen) {
                    seen = R;
                    A = m + 1;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const int Ap = __shfl_up_sync(FULL, A, d);
                        if (lane - d >= start) A = max(A, Ap + d);
                    }
                }
                const int in = __shfl_sync(FULL, vin, 0);
                const bool hang = start == 0 && cin;  // the segment hangs on the row before the warp
                if (!done && (R & need) == need && (!hang || in != 0)) {
                    const int l = hang ? max(A, in + lane + 1) : A;
                    lv[tid] = l;
                    st_relaxed(level + r, l);
                    my_max = max(my_max, l);
                    done = true;
                }
            } else if (R == FULL) {
                // every row's outside columns are known: one pass in order, each lane final by its turn
                int l = m + 1;
                const unsigned T = __reduce_or_sync(FULL, inmask);
#pragma unroll
                for (int q = 0; q < 31; q++)
                    if (T >> q & 1u) {
                        const int lq = __shfl_sync(FULL, l, q);
                        if (inmask >> q & 1u) l = max(l, lq + 1);
                    }
                if (!done) {
                    lv[tid] = l;
                    st_relaxed(level + r, l);
                    my_max = max(my_max, l);
                }
                break;
            } else {
                if (stalled && R != seen) {
                    // some columns are long in coming: the rows that can be done without them are
                    seen = R;
                    for (unsigned T = __reduce_or_sync(FULL, ready ? inmask : 0u) & R; T; T &= T - 1) {
                        const int q = __ffs(T) - 1;
                        const int lq = __shfl_sync(FULL, inmask == 0 ? m + 1 : 0, q);
                        if (lq != 0 && ready && (inmask >> q & 1u)) {
                            m = max(m, lq);
                            inmask &= ~(1u << q);
                        }
                    }
                }
                if (ready && inmask == 0 && !done) {
                    lv[tid] = m + 1;
                    st_relaxed(level + r, m + 1);
                    my_max = max(my_max, m + 1);
                    done = true;
                }
            }
            if (!__any_sync(FULL, !done)) break;
            all = __any_sync(FULL, again);
            stalled = false;
            if (!all) {
                // nothing to do before some lane's last pending column is known: in natural
                // order the others mostly come before it
                const int hi = 31 - __clz(pend);
                int cc = -1, v = 0;
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (hi == u) cc = c[u];
                for (int k = 0;; k++) {
                    if (cc >= R0) v = lv[cc - R0];
                    else if (cc >= 0) v = ld_relaxed(level + cc);
                    if (__any_sync(FULL, v != 0)) break;
                    if (k == kLvStall && !chain && R != seen) {
                        stalled = true;
                        break;
                    }
                    if ((++it & 63u) == 0 && give_up(t0, st, budget, w0)) {
                        fail = true;
                        break;
                    }
                }
                if (v != 0) {
                    pend &= ~(1u << hi);
                    if (cinbit >> hi & 1u) vin = v;
                    else m = max(m, v);
                }
                all = __any_sync(FULL, v != 0 && pend != 0);
            }
        }
        if (fail) abort_flag = 1;
        __syncthreads();  // the group's levels are read no more
        if (abort_flag) return;
    }
    my_max = __reduce_max_sync(FULL, my_max);
    if (lane == 0 && my_max > 0) atomicMax(nlevs, my_max);
}

__global__ void k_keys(const int* __restrict__ rowptr, const int* __restrict__ level, int n, int* __restrict__ key,
                       int* __restrict__ iota, int* counts, int* longer)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int len = rowptr[i + 1] - rowptr[i] - 1;
        int k = 7 * (level[i] - 1) + bucket_of(len);
        key[i] = k;
        iota[i] = i;
        const unsigned over = __ballot_sync(__activemask(), len > 32);
        if (over && (threadIdx.x & 31) == __ffs(over) - 1) atomicAdd(longer, __popc(over));
        unsigned peers = __match_any_sync(__activemask(), k);
        if ((threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(counts + k, __popc(peers));
    }
}

// Is the matrix a stencil on lines of equal length (lines.cuh)?  stats[16] = the
// length w, 0: no; from the distance of 32 sampled rows to their last column
// that is not the row before.
__global__ void k_line_width(const int* __restrict__ rowptr, const int* __restrict__ col, int n, int* stats)
{
    const int r = (int)((long long)n * (threadIdx.x + 1) / 33);
    int z = rowptr[r + 1] - 2, d = 0;
    if (z >= rowptr[r] && col[z] == r - 1) z--;
    if (z >= rowptr[r]) d = r - col[z];
    const unsigned same = __match_any_sync(0xffffffffu, d);
    const int votes = d ? __popc(same) : 0;
    const int most = __reduce_max_sync(0xffffffffu, votes);
    const unsigned who = __ballot_sync(0xffffffffu, votes == most);
    if (threadIdx.x == __ffs(who) - 1) stats[16] = most >= 16 ? d : 0;
}

// stats[17] |= 1 where a row has more than kLineOff off-diagonals, or one inside
// its chunk of 32 (cut at line starts) beside the row before; stats[18] = the most
// of a row; stats[19] = lines whose first row reads the row before.
__global__ void k_line_check(const int* __restrict__ rowptr, const int* __restrict__ col, int n, int* stats)
{
    const int w = stats[16];
    int most = 0, joined = 0;
    bool bad = w < 32;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n && !bad; r += gridDim.x * blockDim.x) {
        const int p = r % w, c0 = r - p % 32, s = rowptr[r], e = rowptr[r + 1] - 1;
        most = max(most, e - s);
        bad = e - s > kLineOff;
        for (int z = s; z < e && !bad; z++) {
            const int c = col[z];
            if (c == r - 1) joined += p == 0;
            else bad = c >= c0;
        }
    }
    bad = __any_sync(0xffffffffu, bad);
    most = __reduce_max_sync(0xffffffffu, most);
    joined = __reduce_add_sync(0xffffffffu, joined);
    if ((threadIdx.x & 31) == 0) {
        if (bad) stats[17] = 1;
        if (most) atomicMax(stats + 18, most);
        if (joined) atomicAdd(stats + 19, joined);
    }
}

// warps per key (get_warps_per_bucks :66-71 with get_size_from_pos :84-102)
__global__ void k_warps_per_key(const int* __restrict__ counts, int K, int* __restrict__ wpk)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k <= K; k += gridDim.x * blockDim.x) {
        if (k == K) {
            wpk[k] = 0;
            continue;
        }
        int b = k % 7;
        int sz = b == 6 ? 1 : (1 << b);
        wpk[k] = (int)(((long long)counts[k] * sz + 31) / 32);
    }
}

// one thread per multirow warp (kernel_base :244-270)
__global__ void k_warp_map(const int* __restrict__ warp_off, const int* __restrict__ row_off, int K, int n_warps,
                           int n, int* __restrict__ ibase, int* __restrict__ ivect, int* __restrict__ wlev)
{
    for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < n_warps; w += gridDim.x * blockDim.x) {
        int lo = 0, hi = K - 1;  // largest k with warp_off[k] <= w
        while (lo < hi) {
            int mid = (lo + hi + 1) >> 1;
            if (warp_off[mid] <= w) lo = mid;
            else hi = mid - 1;
        }
        int k = lo, b = k % 7;
        int size = b == 6 ? 0 : (1 << b);
        int sz = size == 0 ? 1 : size;
        ibase[w] = row_off[k] + (w - warp_off[k]) * (32 / sz);
        ivect[w] = size;
        wlev[w] = k / 7 + 1;
        if (w == 0) ibase[n_warps] = n;
    }
}

// Sizes and first positions of the levels, and the statistics that
// choose_level_cta reads: stats[c] = sum over the levels past the first of
// ceil(size / (4 << c)) - 1, the steps beyond one of a CTA that takes 4 << c
// rows of a level at once; stats[8 + b] = rows of bucket b; stats[15] = rows
// of more than 32 off-diagonals (k_keys).
__global__ void k_level_sizes(const int* __restrict__ counts, const int* __restrict__ row_off, int nlevs,
                              int* __restrict__ lev_size, int* __restrict__ lptr, int* stats)
{
    __shared__ int acc[16];
    if (threadIdx.x < 16) acc[threadIdx.x] = 0;
    __syncthreads();
    for (int l = blockIdx.x * blockDim.x + threadIdx.x; l <= nlevs; l += gridDim.x * blockDim.x) {
        lptr[l] = row_off[7 * l];  // row_off[7 * nlevs] = n
        if (l == nlevs) break;
        int s = 0;
        for (int b = 0; b < 7; b++) {
            const int k = counts[7 * l + b];
            s += k;
            if (k) atomicAdd(acc + 8 + b, k);
        }
        lev_size[l] = s;
        if (l > 0)
            for (int c = 0; c < 8; c++) {
                const int extra = (s - 1) >> (2 + c);
                if (extra) atomicAdd(acc + c, extra);
            }
    }
    __syncthreads();
    if (threadIdx.x < 16 && acc[threadIdx.x]) atomicAdd(stats + threadIdx.x, acc[threadIdx.x]);
}

__global__ void k_inverse(const int* __restrict__ perm, int n, int* __restrict__ inv)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) inv[perm[k]] = k;
}



struct Place {
    int** p;
    long long ints;
};

// Device arrays, in one allocation or one each (share_block); the allocations are
// added to blocks.
cudaError_t place(std::vector<int*>& blocks, long long small, std::initializer_list<Place> arrays)
{
    std::vector<long long> ints;
    long long sum = 0;
    for (const Place& a : arrays) {
        ints.push_back(std::max<long long>(1, a.ints));
        sum += block_part(ints.back());
    }
    const bool share = share_block(ints.data(), (int)ints.size(), small);
    int* at = nullptr;
    int k = 0;
    for (const Place& a : arrays) {
        const long long n = block_part(ints[k++]);
        if (!at) {
            cudaError_t e = dalloc(&at, share ? sum : n);
            if (e != cudaSuccess) return e;
            blocks.push_back(at);
        }
        *a.p = at;
        at = share ? at + n : nullptr;
    }
    return cudaSuccess;
}

}  // namespace

// Checks a device CSR; returns 0, SPTRSV_ERR_INVALID_CSR (with *bad_row) or a CUDA error code.
// d_res: two device ints of scratch.
int validate_csr_device(const int* rowptr, const int* col, int n, int nnz, int* d_res, cudaStream_t s, int* bad_row)
{
    *bad_row = -1;
    if (n <= 0) return 0;
    int h[2] = {0, 0x7fffffff};
    cudaError_t e = cudaMemcpyAsync(d_res, h, sizeof(h), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        k_validate<<<grid_for(n, 256), 256, 0, s>>>(rowptr, col, n, nnz, d_res);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, d_res, sizeof(h), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(e, "validate_csr_device");
    if (h[0]) {
        *bad_row = h[1];
        return SPTRSV_ERR_INVALID_CSR;
    }
    return 0;
}

// Runs the whole analysis; fills *info per `mode` and registers the record.
int run_analysis_impl(dfr_analysis_info_t* info, const sp_mat_t* L, MODE mode, const LevelTasks* tasks)
{
    if (!info || !L) return set_error(SPTRSV_ERR_INVALID_ARG, "analysis: NULL info or matrix");
    const int n = L->nr;
    if (n < 0 || L->nc != n || L->nnz < n) return set_error(SPTRSV_ERR_INVALID_ARG, "analysis: bad sizes n=%d nnz=%d", n, L->nnz);
    if (n > 0 && (!L->ia || !L->ja)) return set_error(SPTRSV_ERR_INVALID_ARG, "analysis: NULL device arrays");
    Ctx* c = ctx();
    if (!c) return set_error(SPTRSV_ERR_CUDA, "analysis: no CUDA device");
    cudaStream_t s = 0;
    const int nnz = L->nnz;

    AnalysisRec* rec = new AnalysisRec();
    rec->device = c->device;
    rec->n = n;
    rec->nnz = nnz;
    std::vector<int*> scratch;  // its allocations
    auto fail = [&](int code) {
        free_blocks(scratch);
        free_blocks(rec->slab);
        delete rec;
        return code;
    };
#define ACHK(call)                                              \
    do {                                                        \
        cudaError_t e_ = (call);                                \
        if (e_ != cudaSuccess) return fail(cuda_fail(e_, #call)); \
    } while (0)
    int *d_rowctr, *d_iorder, *d_inv, *d_key, *d_key2, *d_val2, *d_scr;
    ACHK(place(rec->slab, kRowShare, {{&d_rowctr, n + 64LL}, {&d_iorder, n}, {&d_inv, n}}));
    rec->d_levels = d_rowctr + 64;
    const long long scr = block_part(radix_scratch_ints(n));
    ACHK(place(scratch, kRowShare, {{&d_key, n}, {&d_key2, n}, {&d_val2, n}, {&d_scr, scr + 64}}));
    int* d_nlevs = d_scr + scr;

    // 0. validation (the status block must be clean before the bounded waits)
    {
        int e = sync_status(s);
        if (e) return fail(e);
        int bad = -1;
        e = validate_csr_device(L->ia, L->ja, n, nnz, d_nlevs + 2, s, &bad);
        if (e) fail(e);
        if (e == SPTRSV_ERR_INVALID_CSR)
            return set_error(e, "analysis: row %d is not lower-triangular CSR with sorted columns and the diagonal last",
                             bad);
        if (e) return e;
    }
    ACHK(cudaMemsetAsync(rec->d_levels, 0, sizeof(int) * (size_t)(n > 0 ? n : 1), s));
    ACHK(cudaMemsetAsync(d_nlevs, 0, sizeof(int), s));
    ACHK(cudaMemsetAsync(d_rowctr, 0, sizeof(int), s));

    // 1. levels
    int nlevs = 0;
    if (n > 0) {
        const long long nt = tasks ? tasks->n : ((long long)n + kLvGroup - 1) / kLvGroup;
        // columns per lane and poll round: 4 covers a stencil's row at once
        auto kern = (long long)nnz - n <= 4LL * n ? k_levels<4> : k_levels<8>;
        ACHK(launch_persistent(kern, kLvGroup, 0, nt, s, L->ia, L->ja, n, rec->d_levels, d_nlevs, c->d_status, wait_budget_ns(), tasks ? tasks->r0 : (const int*)nullptr,
                               tasks ? tasks->cnt : (const int*)nullptr, nt));
        ACHK(cudaMemcpyAsync(&nlevs, d_nlevs, sizeof(int), cudaMemcpyDeviceToHost, s));
        int st = sync_status(s);
        if (st) return fail(st);
    }
    rec->nlevs = nlevs;
    const long long K = 7LL * nlevs;

    // 2-3. keys, counts, stable sort
    int *d_levsz, *d_stats;
    ACHK(place(rec->slab, kOtherShare,
               {{&rec->d_counts, K + 1}, {&d_levsz, nlevs + 1LL}, {&rec->d_lptr, nlevs + 1LL}, {&d_stats, 64}}));
    ACHK(cudaMemsetAsync(rec->d_counts, 0, sizeof(int) * (size_t)(K + 1), s));
    ACHK(cudaMemsetAsync(d_stats, 0, sizeof(rec->stats), s));
    if (n > 0) {
        k_keys<<<grid_for(n, 256), 256, 0, s>>>(L->ia, rec->d_levels, n, d_key, d_iorder, rec->d_counts, d_stats + 15);
        ACHK(cudaGetLastError());
        k_line_width<<<1, 32, 0, s>>>(L->ia, L->ja, n, d_stats);
        ACHK(cudaGetLastError());
        k_line_check<<<grid_for(n, 256), 256, 0, s>>>(L->ia, L->ja, n, d_stats);
        ACHK(cudaGetLastError());
        ACHK(radix_sort_pairs(d_key, d_iorder, d_key2, d_val2, n, (int)(K - 1), d_scr, s));
    }

    // 4. multirow warp map (always built; exposed in info for MULTIROW/ALL),
    // its scratch where the sort's keys were unless there are more keys than rows
    int *d_wpk = d_key, *d_rowoff = d_key2, *d_scr2 = d_val2;
    bool fits = K + 1 <= n;
    if (scratch.size() == 1) {  // the three arrays are one stretch
        const long long pk = block_part(K + 1);
        fits = 2 * pk + block_part(scan_scratch_ints(K + 1)) <= 3 * block_part(n);
        d_rowoff = d_wpk + pk;
        d_scr2 = d_rowoff + pk;
    }
    if (!fits) {
        free_blocks(scratch);
        ACHK(place(scratch, kOtherShare, {{&d_wpk, K + 1}, {&d_rowoff, K + 1}, {&d_scr2, scan_scratch_ints(K + 1)}}));
    }
    int n_warps = 0;
    if (K > 0) {
        k_warps_per_key<<<grid_for(K + 1, 256), 256, 0, s>>>(rec->d_counts, (int)K, d_wpk);
        ACHK(cudaGetLastError());
        ACHK(scan_exclusive(d_wpk, d_wpk, K + 1, d_scr2, s));
        ACHK(scan_exclusive(rec->d_counts, d_rowoff, K + 1, d_scr2, s));
        k_level_sizes<<<grid_for(nlevs + 1LL, 256), 256, 0, s>>>(rec->d_counts, d_rowoff, nlevs, d_levsz, rec->d_lptr,
                                                                 d_stats);
        ACHK(cudaGetLastError());
        ACHK(cudaMemcpyAsync(rec->stats, d_stats, sizeof(rec->stats), cudaMemcpyDeviceToHost, s));
        ACHK(cudaMemcpyAsync(&n_warps, d_wpk + K, sizeof(int), cudaMemcpyDeviceToHost, s));
        ACHK(cudaStreamSynchronize(s));
    }
    rec->n_warps = n_warps;
    ACHK(place(rec->slab, kOtherShare, {{&rec->d_ibase, n_warps + 1LL}, {&rec->d_ivect, n_warps}, {&rec->d_wlev, n_warps}}));
    if (n_warps > 0) {
        k_warp_map<<<grid_for(n_warps, 256), 256, 0, s>>>(d_wpk, d_rowoff, (int)K, n_warps, n, rec->d_ibase,
                                                           rec->d_ivect, rec->d_wlev);
        ACHK(cudaGetLastError());
    } else {
        ACHK(cudaMemsetAsync(rec->d_ibase, 0, sizeof(int), s));
    }

    // extras the reference declares but never fills
    if (n > 0) {
        k_inverse<<<grid_for(n, 256), 256, 0, s>>>(d_iorder, n, d_inv);
        ACHK(cudaGetLastError());
    }
    ACHK(cudaStreamSynchronize(s));
    free_blocks(scratch);
#undef ACHK

    info->mode = mode;
    info->lev_ctr = 0;
    info->nlevs = nlevs;
    info->lev_size = d_levsz;
    info->inv_iorder = d_inv;
    info->iorder = d_iorder;
    info->row_ctr = d_rowctr;
    if (mode == MULTIROW || mode == ALL) {
        info->n_warps = n_warps;
        info->ibase_row = rec->d_ibase;
        info->ivect_size_warp = rec->d_ivect;
        info->warp_lev = rec->d_wlev;
        rec->map_in_info = true;
    } else {
        info->n_warps = 0;
        info->ibase_row = nullptr;
        info->ivect_size_warp = nullptr;
        info->warp_lev = nullptr;
        rec->map_in_info = false;
    }
    register_analysis(d_rowctr, rec);
    return ok();
}

}  // namespace sptrsv
