// level_cta.cuh — narrow systems solved level by level by one CTA.
//
// Where levels hold few rows a solve is as long as its levels are many, and a
// level that hands its values on through L2 costs 0.8-0.95 us (a hop of 707
// cycles from one SM's store to another's poll, and the work around it).
// Here one CTA solves the whole system: x lives in shared memory, and the
// hop from level to level is a named barrier (about 25 cycles).
//
// The CTA's 16 warps form NT = 16 / G teams of G warps, and team t takes the
// levels t, t + NT, ...  The chain of dependent loads that a row needs (level
// bounds, row, range, entries, their columns' positions) runs five turns
// ahead, a link a turn, so no turn waits for two of them.  Between two levels
// only this is left: barrier, shared-memory loads of x, products, lane
// reduction, one shared-memory store, arrival at the next team's barrier.
// Barrier t carries the hand-over to team t: the G warps of the level before
// arrive, the team's G warps wait.  Its next use, NT levels later, comes after
// every level between, so the 16 hardware barriers serve any number of levels,
// and no wait depends on another CTA.
//
// Bound: that chain, 230 cycles a level (n = 2e4 in a band of 16, G = 1) to
// 320 (n = 1e5 in a band of 256, G = 2), and with few large teams the turn
// itself (about 1,600 cycles, the issue slots of 16 warps).  Before and after,
// FP64 drop-in solves: banded n = 1e5 5.9 -> 1.0 ms, n = 5000 645 -> 105 us,
// n = 3e4 in a band of 16 16.4 -> 3.2 ms, 61 x 47 grid 88 -> 17 us.
//
// Arithmetic per row as in k_sptrsv: lane sl of a row's kp lanes takes the
// entries sl, sl + kp, ... in order, then a shuffle reduction; rows of the
// first level (no off-diagonals) are b / diag or b * (1 / diag) as there.
//
// x in shared memory: all of it when it fits (slot = row), else a ring over
// the level order (slot = position mod ring, RING): a column whose position
// lies more than the ring before the end of the level is read from x in
// global memory, where the rows were stored before the barrier.
#pragma once

#include "solve_kernels.cuh"

namespace sptrsv {

constexpr int kTeamWarps = 16;  // NT = 16 / G teams, one hardware barrier each
constexpr int kTeamU = 4;       // entries per lane loaded ahead

struct LevelCta {
    const int* __restrict__ lptr;  // [nlevs + 1] first position of each level
    const int* __restrict__ inv;   // row -> position (RING)
    int nlevs;
    int slots;   // RING: ring slots (a power of two); else n.  Slot `slots` holds 0 for unused entries
    int divide;  // first level: b / diag
};

// What is known of a lane's row, a stage further each turn of its team.
struct TeamRow {
    int pos, end;  // position of the row, end of its level; pos >= end: no row
    int r, s, e;   // row, its off-diagonal range
};
template <typename T>
struct TeamEnt {
    int c[kTeamU];
    T v[kTeamU];
    T d;  // 1 / diag, or the diagonal (M::kInvStored)
    T b;
};

template <class M, typename T, typename BT, int OUT, int KP, bool RING>
__global__ void __launch_bounds__(32 * kTeamWarps, 1) k_sptrsv_level_cta(M m, LevelCta lc, int G, const BT* __restrict__ b, T* x,
                                                            double* x64)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    volatile T* xs = reinterpret_cast<volatile T*>(smem_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int NT = kTeamWarps / G, team = warp / G, sub = warp - team * G;
    const int next = team + 1 == NT ? 0 : team + 1;
    constexpr int RPS = 32 / KP;  // rows per step of a warp
    const int first = sub * RPS + lane / KP, sl = lane % KP;
    const int zero = lc.slots, mask = lc.slots - 1;
    auto own_slot = [&](int r, int pos) { return RING ? (pos & mask) : r; };
    auto publish64 = [&](int r, T v) {
        if (OUT == OUT_SET64) x64[r] = (double)publishable(v);
        if (OUT == OUT_ADD64) x64[r] += (double)publishable(v);
    };

    // first level: rows without off-diagonals, all warps
    const int n0 = __ldg(lc.lptr + 1);
    for (int pos = threadIdx.x; pos < n0; pos += blockDim.x) {
        const RowRef q = m.row(pos);
        const T v = lc.divide ? (T)b[q.r] / (T)m.diag(q) : (T)b[q.r] * (T)m.inv(q);
        xs[own_slot(q.r, pos)] = v;
        x[q.r] = publishable(v);
        publish64(q.r, v);
    }
    if (threadIdx.x == 0) xs[zero] = (T)0;
    __syncthreads();

    // the stages of the rows to come: level bounds, row, range, entries, slots
    TeamRow w1, w2, w3, cur;
    TeamEnt<T> e3, ec;
    int pc[kTeamU];  // RING: positions of the current row's columns
    int a0 = 0, z0 = 0;
    w1.pos = w2.pos = w3.pos = cur.pos = 0;
    w1.end = w2.end = w3.end = cur.end = 0;
#pragma unroll
    for (int u = 0; u < kTeamU; u++) pc[u] = 0;
    for (int l = 1 + team - 5 * NT; l < lc.nlevs; l += NT) {
        if (l >= 1) {
            // everything that does not depend on the levels before
            const bool act = cur.pos < cur.end, mine = act && sl == 0;
            const int n = act ? max(0, (cur.e - cur.s - sl + KP - 1) / KP) : 0;
            int cc[kTeamU];
            T vv[kTeamU];
            bool far = false;
#pragma unroll
            for (int u = 0; u < kTeamU; u++) {
                cc[u] = zero;
                vv[u] = (T)0;
                if (u < n) {
                    vv[u] = -ec.v[u];
                    if (!RING) cc[u] = ec.c[u];
                    else if (cur.end - pc[u] <= lc.slots) cc[u] = pc[u] & mask;
                    else far = true;
                }
            }
            const T piv = act ? (M::kInvStored ? ec.d : (T)1 / ec.d) : (T)0;
            const T rhs = mine ? ec.b : (T)0;
            const int p1 = cur.pos - first + (sub + G) * RPS;  // this warp's next rows of the level (uniform)
            const bool plain = __all_sync(0xffffffffu, n <= kTeamU && !far && p1 >= cur.end);
            const int own = own_slot(cur.r, cur.pos);
            if (l > 1) asm volatile("barrier.cta.sync %0, %1;" ::"r"(team), "r"(64 * G) : "memory");
            T xv[kTeamU];
#pragma unroll
            for (int u = 0; u < kTeamU; u++) xv[u] = xs[cc[u]];
            auto sum = [&]() {
                T s0 = rhs, s1 = vv[1] * xv[1];
                s0 += vv[0] * xv[0];
                s1 += vv[3] * xv[3];
                s0 += vv[2] * xv[2];
                return s0 + s1;
            };
            T acc = sum();
            if (plain) {
#pragma unroll
                for (int o = KP >> 1; o >= 1; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o, KP);
                const T v = acc * piv;
                if (mine) xs[own] = v;
                if (RING && mine) x[cur.r] = publishable(v);  // read there once it has left the ring
                if (l + 1 < lc.nlevs)
                    asm volatile("barrier.cta.arrive %0, %1;" ::"r"(next), "r"(64 * G) : "memory");
                if (!RING && mine) x[cur.r] = publishable(v);
                if (mine) publish64(cur.r, v);
            } else {
                if (RING) {  // columns that left the ring long ago (summed anew: an infinity times the 0 above is NaN)
#pragma unroll
                    for (int u = 0; u < kTeamU; u++)
                        if (u < n && cc[u] == zero) xv[u] = ld_relaxed(x + ec.c[u]);
                    if (far) acc = sum();
                }
                auto rest = [&](int p, int e) {  // entries beyond the ones loaded ahead
                    T t = (T)0;
                    for (; p < e; p += KP) {
                        const int c = m.c(p);
                        int k = c;
                        if (RING) {
                            const int q = __ldg(lc.inv + c);
                            k = cur.end - q <= lc.slots ? (q & mask) : -1;
                        }
                        t -= (T)m.v(p) * (k >= 0 ? (T)xs[k] : ld_relaxed(x + c));
                    }
                    return t;
                };
                if (n > kTeamU) acc += rest(cur.s + sl + kTeamU * KP, cur.e);
#pragma unroll
                for (int o = KP >> 1; o >= 1; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o, KP);
                const T v = acc * piv;
                if (mine) {
                    xs[own] = v;
                    x[cur.r] = publishable(v);
                    publish64(cur.r, v);
                }
                for (int p0 = p1; p0 < cur.end; p0 += G * RPS) {  // levels wider than the team: rows on the spot
                    const int pos = p0 + lane / KP;
                    T t = (T)0, pv = (T)0;
                    RowRef q;
                    if (pos < cur.end) {
                        q = m.row(pos);
                        pv = (T)m.inv(q);
                        t = (sl == 0 ? (T)b[q.r] : (T)0) + rest(q.s + sl, q.e);
                    }
#pragma unroll
                    for (int o = KP >> 1; o >= 1; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o, KP);
                    if (pos < cur.end && sl == 0) {
                        const T vw = t * pv;
                        xs[own_slot(q.r, pos)] = vw;
                        x[q.r] = publishable(vw);
                        publish64(q.r, vw);
                    }
                }
                if (l + 1 < lc.nlevs)
                    asm volatile("barrier.cta.arrive %0, %1;" ::"r"(next), "r"(64 * G) : "memory");
            }
        }
        // the next level's columns are here: their positions
        cur = w3;
        ec = e3;
        if (RING && cur.pos < cur.end) {
#pragma unroll
            for (int u = 0; u < kTeamU; u++)
                if (cur.s + sl + u * KP < cur.e) pc[u] = __ldg(lc.inv + ec.c[u]);
        }
        // the range of the row after it is here: its entries
        w3 = w2;
        if (w3.pos < w3.end) {
#pragma unroll
            for (int u = 0; u < kTeamU; u++) {
                const int p = w3.s + sl + u * KP;
                if (p < w3.e) {
                    e3.c[u] = m.c(p);
                    e3.v[u] = (T)m.v(p);
                }
            }
            e3.d = (T)m.scale(w3.pos, w3.e);
            e3.b = (T)b[w3.r];
        }
        // and so on: range, row, level
        w2 = w1;
        if (w2.pos < w2.end) m.range(w2.pos, w2.r, w2.s, w2.e);
        w1.pos = a0 + first;
        w1.end = z0;
        if (w1.pos < w1.end) w1.r = m.id(w1.pos);
        const int ln = l + 5 * NT;
        a0 = z0 = 0;
        if (ln < lc.nlevs) {
            a0 = __ldg(lc.lptr + ln);
            z0 = __ldg(lc.lptr + ln + 1);
        }
    }
}

}  // namespace sptrsv
