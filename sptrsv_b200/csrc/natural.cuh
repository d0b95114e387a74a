// natural.cuh — solves in natural row order, no analysis needed (SIMPLE, the
// allocation-free solve).
//
// CTA g takes the groups g, g + G, ... of 256 consecutive rows, one thread
// per row.  The group's x lives in shared memory (the sentinel first), so a
// column inside the group is a shared-memory poll; columns of earlier groups
// are polled in x.  Natural order is topological and the CTAs are co-resident,
// so the lowest unfinished row never waits on an unfinished one.
//
// A lane's columns outside its warp are taken kNatU at a time: polled
// together until all are known, then subtracted in their order, so sums do not
// depend on timing.  Columns inside the warp are not polled:
//   * where they are the row before only, with |L_i,i-1 / L_ii| <= 1 (stencils),
//     the warp is a first-order recurrence x_j = a_j + b_j x_j-1, closed by an
//     affine prefix scan over the lanes into which the row before the warp
//     enters last.  Lanes that start a new grid line start a new segment of
//     the scan, and a segment is closed as soon as its own rows are known:
//     one line's end does not hold up the next line's start.  A row is always
//     of the same scan over its segment, whichever rows were known together;
//     rows that are not finite by it are taken one after another;
//   * otherwise one pass over the lanes that are read, in order, broadcasts
//     each value to the rows that read it, once all of the warp's outside
//     columns are known or, as far as it goes, when some are long in coming;
//   * where a row is not sorted there (columns inside the warp that do not
//     ascend, or one outside after one inside), its entries are looked up for
//     every lane in turn.
// Before it looks at all its columns a warp waits for one word, the smallest
// over its rows without a column inside the warp of the row's largest column
// (the line above, where a scan waits for the row before it last): a warp
// far from the front costs one sector a poll.
//
// Bound: the hops.  FP64 solves before and after (a warp took 32 rows one after
// another): 1000 x 900 grid 444 -> 1.2 ms, 101 x 90 x 97 grid 543 -> 0.69 ms,
// Zipf n = 1e6 39.6 -> 2.1 ms, banded n = 1e5 55.5 -> 8.9 ms, dense 32-row
// blocks n = 3e5 74 -> 49 us.
//
// STAGE: the entries of a warp's 32 rows are contiguous in the caller's CSR; up
// to kNatStage of them are copied to shared memory by coalesced cp.async, as
// a lane reading its own row entry by entry costs the load unit 32 sectors an
// entry.
//
// CHECK (for callers whose CSR was never validated on the host): before a
// row's entries are touched, its range must satisfy 0 <= rowptr[r] <
// rowptr[r+1] <= nnz with the diagonal last, and every off-diagonal column
// must satisfy 0 <= c < r before it is used.  A violation records
// SPTRSV_ERR_INVALID_CSR and the row in the status word and the CTA leaves
// without any access through the bad index.
#pragma once

#include "solve_kernels.cuh"

namespace sptrsv {

constexpr int kNatGroup = 256;   // rows (threads) of a group
constexpr int kNatU = 4;         // columns per lane and round
constexpr int kNatStage = 544;   // staged entries of a warp (32 rows of 17)
constexpr int kNatStall = 16;    // polls without an answer after which a warp does what it can

// Dynamic shared memory of the staged form.
template <typename V>
constexpr size_t nat_stage_bytes()
{
    return (size_t)(kNatGroup / 32) * kNatStage * (sizeof(V) + sizeof(int));
}

template <class M, typename T, typename BT, int OUT, bool CHECK, bool STAGE>
__global__ void __launch_bounds__(kNatGroup, 3) k_sptrsv_natural(M m, int n, const BT* __restrict__ b, T* x, double* x64,
                                                             DevStatus* st, unsigned long long budget)
{
    typedef typename M::V V;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ volatile T xs[kNatGroup];
    __shared__ int abort_flag;
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
    const unsigned upto = FULL >> (31 - lane);  // lanes 0..lane
    V* sval = reinterpret_cast<V*>(smem_raw) + wib * kNatStage;
    int* scol = reinterpret_cast<int*>(smem_raw + (size_t)(kNatGroup / 32) * kNatStage * sizeof(V)) + wib * kNatStage;
    if (tid == 0) abort_flag = 0;
    const int ngroups = (n + kNatGroup - 1) / kNatGroup;
    for (int g = blockIdx.x; g < ngroups; g += gridDim.x) {
        const int R0 = g * kNatGroup, r = R0 + tid, w0 = R0 + wib * 32;
        const bool act = r < n;
        xs[tid] = sentinel_value<T>();
        RowRef q;
        q.r = r;
        q.s = q.e = q.d = 0;
        bool fail = false;
        if (act) q = m.row(r);
        if constexpr (CHECK) {
            const bool bad = act && (!(q.s >= 0 && q.s <= q.e && q.e < m.nnz) || m.c(q.e) != q.r);
            if (bad) {
                report(st, SPTRSV_ERR_INVALID_CSR, q.r);
                q.s = q.e = 0;
            }
            fail = __any_sync(FULL, bad);
        }
        int base = 0;
        bool staged = false;
        if constexpr (STAGE) {
            const int end = __reduce_max_sync(FULL, act ? q.e : 0);  // one past the warp's last off-diagonal
            base = __shfl_sync(FULL, q.s, 0);
            staged = end - base <= kNatStage;
            if (staged) {
                for (int i = lane; i < end - base; i += 32) {
                    cp_async_ca(scol + i, m.col + base + i);
                    cp_async_ca(sval + i, m.val + base + i);
                }
            }
        }
        T acc = (T)0, piv = (T)0;
        if (act && !fail) {
            acc = (T)b[q.r];
            piv = (T)m.inv(q);
        }
        if constexpr (STAGE) {
            cp_async_wait_all();
            __syncwarp();
        }
        auto col_at = [&](int p) -> int { return STAGE && staged ? scol[p - base] : m.c(p); };
        auto val_at = [&](int p) -> T { return (T)(STAGE && staged ? sval[p - base] : m.v(p)); };

        int p = q.s, nb = 0, c[kNatU];
        T v[kNatU], xv[kNatU];
        unsigned pend = 0;      // columns of the round outside the warp, not known yet
        unsigned outside = 0;   // columns of the round outside the warp
        unsigned inmask = 0;    // lanes of this warp whose values the row reads and has not got
        int pin = 0x7fffffff, lastin = -1;  // the row's first entry inside the warp; the last such column
        bool odd = false;
        auto round = [&]() -> bool {  // false: a bad column (CHECK)
            nb = min(kNatU, q.e - p);
            outside = 0;
            bool good = true;
#pragma unroll
            for (int u = 0; u < kNatU; u++) {
                c[u] = -1;
                v[u] = (T)0;
                if (u < nb) {
                    c[u] = col_at(p + u);
                    v[u] = val_at(p + u);
                    if (CHECK && (c[u] < 0 || c[u] >= q.r)) {
                        report(st, SPTRSV_ERR_INVALID_CSR, q.r);
                        good = false;
                    } else if (c[u] >= w0) {
                        inmask |= 1u << (c[u] - w0);
                        odd |= c[u] <= lastin;
                        lastin = c[u];
                        pin = min(pin, p + u);
                    } else {
                        outside |= 1u << u;
                        odd |= lastin >= 0;
                    }
                }
            }
            pend = outside;
            // the rest of a row that has come inside the warp is inside, when it is sorted
            if (good && pin < q.e)
                for (int z = p + nb; z < q.e; z++, nb++) {
                    const int cc = col_at(z);
                    if (CHECK && (cc < 0 || cc >= q.r)) {
                        report(st, SPTRSV_ERR_INVALID_CSR, q.r);
                        good = false;
                        break;
                    }
                    if (cc < w0) {
                        odd = true;
                        break;
                    }
                    inmask |= 1u << (cc - w0);
                    odd |= cc <= lastin;
                    lastin = cc;
                }
            return good;
        };
        if (!round()) fail = true;
        if (CHECK) fail = __any_sync(FULL, fail);

        const bool sub = lane > 0 && (inmask >> (lane - 1) & 1u);
        T lsub = (T)0, beta = (T)0;  // the row before: its entry, its factor where the recurrence continues it
        unsigned cinbit = 0;  // lane 0: the column that is the row before the warp
        int far = -1;
#pragma unroll
        for (int u = 0; u < kNatU; u++)
            if (u < min(nb, kNatU) && c[u] == r - 1) {
                lsub = v[u];
                beta = -lsub * piv;
                if (lane == 0) cinbit = 1u << u;
            }
        const bool single = __popc(inmask) == (q.e - p - __popc(outside));  // no column inside the warp twice
        const bool chain = __all_sync(FULL, q.e - p <= kNatU && inmask == (sub ? 1u << (lane - 1) : 0u) && single &&
                                          fabs((double)beta) <= 1.0 && __popc(cinbit) <= 1);
        if (!chain) cinbit = 0;
#pragma unroll
        for (int u = 0; u < kNatU; u++)
            if ((pend & ~cinbit) >> u & 1u) far = max(far, c[u]);
        const bool cin = __shfl_sync(FULL, cinbit, 0) != 0;
        int word = __reduce_min_sync(FULL, act && inmask == 0 ? (cinbit ? w0 - 1 : far) : 0x7fffffff);
        if (cin && word == w0 - 1) {
            const int above = __reduce_min_sync(FULL, far >= 0 ? far : 0x7fffffff);
            if (above != 0x7fffffff) word = above;
        }
        __syncthreads();  // xs is filled
        unsigned it = 0, seen = 0;
        unsigned long long t0 = 0;
        if (!fail && word >= 0 && word != 0x7fffffff)
            while (is_pending(word >= R0 ? (T)xs[word - R0] : ld_relaxed(x + word)))
                if ((++it & 63u) == 0 && give_up(t0, st, budget, w0)) {
                    fail = true;
                    break;
                }

        bool done = !act, ready = !act;  // ready: the columns outside the warp are subtracted
        T A = (T)0, B = (T)0, vin = (T)0;
        bool have_in = false;  // lane 0: the row before the warp is known
        const unsigned S = __ballot_sync(FULL, !sub) | 1u;
        const int start = 31 - __clz(S & upto);
        const unsigned need = upto & (FULL << start);
        // the entries inside the warp, in order: the next one's lane and value, and the one after (at pi)
        int pi = 0x7fffffff, nl = 99, nl2 = 99;
        T nv = (T)0, nv2 = (T)0;
        auto next_in = [&]() {
            nl = nl2;
            nv = nv2;
            nl2 = 99;
            if (++pi < q.e) {
                nl2 = col_at(pi) - w0;
                nv2 = val_at(pi);
            }
        };
        auto finish = [&](T val) {
            val = publishable(val);
            xs[tid] = val;
            publish<T, OUT>(x, x64, (size_t)q.r, val);
            done = true;
            if (chain) return;  // later scans of the warp take the row as this one did
            acc = val;          // what the rows inside the warp that read it take
            piv = (T)1;
            nl = 99;
        };
        bool all = true, stalled = false, walking = false;
        while (!fail) {
            if (all) {
#pragma unroll
                for (int u = 0; u < kNatU; u++)
                    if ((pend >> u & 1u) && c[u] < R0) xv[u] = ld_relaxed(x + c[u]);
#pragma unroll
                for (int u = 0; u < kNatU; u++)
                    if ((pend >> u & 1u) && c[u] >= R0) xv[u] = xs[c[u] - R0];
#pragma unroll
                for (int u = 0; u < kNatU; u++)
                    if ((pend >> u & 1u) && !is_pending(xv[u])) pend &= ~(1u << u);
            }
            bool again = false;
            if (!ready && (pend & ~cinbit) == 0) {
#pragma unroll
                for (int u = 0; u < kNatU; u++)
                    if ((outside & ~cinbit) >> u & 1u) acc -= v[u] * xv[u];
                p += nb;
                if (p < q.e) {
                    if (!round()) fail = true;
                    again = true;
                } else {
                    ready = true;
                }
            }
            if (CHECK) {
                fail = __any_sync(FULL, fail);
                if (fail) break;
            }
            const unsigned R = __ballot_sync(FULL, ready);
            if (chain) {
                if (cinbit && !have_in && (pend & cinbit) == 0) {
                    have_in = true;
#pragma unroll
                    for (int u = 0; u < kNatU; u++)
                        if (cinbit >> u & 1u) vin = xv[u];
                }
                if (R != seen) {
                    seen = R;
                    A = acc * piv;
                    B = beta;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const T Ap = __shfl_up_sync(FULL, A, d), Bp = __shfl_up_sync(FULL, B, d);
                        if (lane - d >= start) {
                            A = A + B * Ap;
                            B = B * Bp;
                        }
                    }
                }
                const bool known = __shfl_sync(FULL, (int)have_in, 0) != 0;
                const T in = __shfl_sync(FULL, vin, 0);
                const bool hang = start == 0 && cin;  // the segment hangs on the row before the warp
                const bool now = !done && (R & need) == need && (!hang || known);
                const T val = hang ? A + B * in : A;  // of the same scan whatever other rows were ready
                T fin = val;
                if (__any_sync(FULL, now && !isfinite(val))) {
                    // such rows one after another, as infinities and NaN spread in substitution; a
                    // row whose scan is finite has only finite ones before it in its segment
                    T t = in;
                    for (int k = 0; k < 32; k++) {
                        if (lane == k) {
                            if (done) fin = xs[tid];
                            else if (!isfinite(val)) fin = publishable((sub || cinbit ? acc - lsub * t : acc) * piv);
                        }
                        t = __shfl_sync(FULL, fin, k);
                    }
                }
                if (now) finish(fin);
            } else {
                const bool full = R == FULL;
                if (full || (stalled && R != seen)) {
                    seen = R;
                    if (ready && !done && !walking) {
                        walking = true;
                        if (!odd && pin < q.e) {
                            pi = pin - 1;
                            next_in();
                            next_in();
                        }
                    }
                    const unsigned T0 = __reduce_or_sync(FULL, ready && !done ? inmask : 0u) & R;
                    if (__any_sync(FULL, odd)) {
                        if (full)
                            for (int k = 0; k < 31; k++)
                                if (T0 >> k & 1u) {
                                    const T xk = __shfl_sync(FULL, acc * piv, k);
                                    if (!done && lane > k && (inmask >> k & 1u))
                                        for (int z = pin; z < q.e; z++)
                                            if (col_at(z) == w0 + k) acc -= val_at(z) * xk;
                                }
                    } else if (full) {
#pragma unroll
                        for (int k = 0; k < 31; k++)
                            if (T0 >> k & 1u) {
                                const T xk = __shfl_sync(FULL, acc * piv, k);
                                if (nl == k) {
                                    acc -= nv * xk;
                                    next_in();
                                }
                            }
                    } else {  // only rows whose columns inside the warp are all final hand on their value
                        for (unsigned Q = T0; Q; Q &= Q - 1) {
                            const int k = __ffs(Q) - 1;
                            const T xk = __shfl_sync(FULL, acc * piv, k);
                            const int fin = __shfl_sync(FULL, (int)(ready && nl == 99), k);
                            if (fin && ready && nl == k) {
                                acc -= nv * xk;
                                inmask &= ~(1u << k);  // not again, should the warp turn out to hold an odd row
                                next_in();
                            }
                        }
                    }
                    if (!done && (full || (ready && nl == 99 && !odd))) finish(acc * piv);
                } else if (!done && ready && inmask == 0) {
                    finish(acc * piv);
                }
            }
            if (!__any_sync(FULL, !done)) break;
            all = __any_sync(FULL, again);
            stalled = false;
            if (!all) {
                // nothing to do before some lane's last pending column is known: in natural
                // order the others mostly come before it
                const int hi = 31 - __clz(pend);
                int cc = -1;
#pragma unroll
                for (int u = 0; u < kNatU; u++)
                    if (hi == u) cc = c[u];
                T got = sentinel_value<T>();
                for (int k = 0;; k++) {
                    if (cc >= R0) got = xs[cc - R0];
                    else if (cc >= 0) got = ld_relaxed(x + cc);
                    if (__any_sync(FULL, !is_pending(got))) break;
                    if (k == kNatStall && !chain && R != seen) {
                        stalled = true;
                        break;
                    }
                    if ((++it & 63u) == 0 && give_up(t0, st, budget, w0)) {
                        fail = true;
                        break;
                    }
                }
                if (cc >= 0 && !is_pending(got)) {
                    pend &= ~(1u << hi);
#pragma unroll
                    for (int u = 0; u < kNatU; u++)
                        if (hi == u) xv[u] = got;
                }
                all = __any_sync(FULL, cc >= 0 && !is_pending(got) && pend != 0);
            }
        }
        if (fail) abort_flag = 1;
        __syncthreads();  // the group's x is read no more
        if (abort_flag) return;
    }
}

}  // namespace sptrsv
