// band.cu — the BAND schedule: one CTA per independent unit of rows, its
// steps handed from warp to warp, x in shared-memory slots.
//
// A unit is a set of consecutive rows that depends on no row outside it:
// the whole matrix, or one block of a partitioned plan's block system.  One
// CTA solves its unit alone, so no flag, poll or wait on another CTA exists
// anywhere.  The unit's rows are cut into steps of at most 32/kp rows with kp
// lanes per row (at most U = 4 entries per lane), every row after the steps of
// the rows it reads, and step t is warp t mod 8's.  While the others work on
// the steps before, a warp has its next two steps' records and its next
// step's right-hand sides on their way into registers; between two steps only
// this is left: a named barrier (about 25 cycles), shared-memory loads of x,
// products, lane reduction, one shared-memory store, arrival at the next
// warp's barrier.  It suits units whose levels are narrow (banded matrices:
// about 16 rows per level).
//
// Bound: that chain, as many times as the unit has steps: 240 cycles a step,
// against 390-480 when one warp took the steps and their records by itself
// (unpacking a record and issuing the next one's loads stood between its
// steps).  Steps are filled by list scheduling: of the rows that are ready,
// those with the longest chain of readers first, whatever their level, so a
// level of 17 rows does not cost two steps.  Banded n = 1e5 (8 in 256) over
// 128 blocks: 153 -> 82 us, whole: 1.80 -> 0.99 ms.
//
// Records.  Step t is one fixed-size record holding, per lane, a packet of
// 16-byte pieces stored piece-major (see band_rec_bytes): the lane's 4 entry
// values and their columns' slots (slot R holds a constant 0 for unused
// entries), the slot of the lane's row, the row of b and x it takes (-1:
// none), whether x is written (a warm-up row's is not), 1 / L_rr and the
// step's kp.  A lane reads its packet with 3-4 coalesced 128-bit loads.
//
// Slots.  A row's value lives in a shared-memory slot from its step until
// the last step that reads it.  The builder hands slots out in step order from
// a free list and takes a slot back after its occupant's last reader (interval
// allocation), so R = the most values alive at once (at most 8192); slot R
// holds 0 for unused entries.  Where list scheduling keeps more than that
// alive, or needs more steps, the steps follow the levels (band_steps.h).
#include <algorithm>
#include <cstring>
#include <exception>
#include <system_error>
#include <thread>
#include <vector>

#include "band_steps.h"
#include "internal.h"
#include "plan.h"
#include "solve_kernels.cuh"

namespace sptrsv {

namespace {

constexpr int kBandWarps = 8;     // one hardware barrier each

// Record of one step: per lane a packet of 16-byte pieces, stored piece-major
// (piece k of lane j at k * 512 + j * 16), so a warp reads a piece with one
// coalesced 128-bit load per lane.
//   FP64 (4 pieces): {v0, v1} {v2, v3} {slot0|slot1, slot2|slot3, os|kp<<16|write<<24, row} {inv, 0}
//   FP32 (3 pieces): {v0..v3} {slot0|slot1, slot2|slot3, os|kp<<16|write<<24, row} {inv, 0, 0, 0}
// (slots and os 16 bits each; kp is the step's, the same in every lane)
__host__ __device__ constexpr int band_pieces(int tsz) { return tsz == 8 ? 4 : 3; }
__host__ __device__ constexpr int band_rec_bytes(int tsz) { return band_pieces(tsz) * 512; }

// One step's record pieces of this lane.
template <typename T>
struct BandRec {
    static constexpr int NP = sizeof(T) == 8 ? 4 : 3, META = NP - 2;
    uint4 c[NP];
    __device__ __forceinline__ void fetch(const unsigned char* r, int lane)
    {
        const uint4* p = reinterpret_cast<const uint4*>(r) + lane;
#pragma unroll
        for (int k = 0; k < NP; k++) c[k] = __ldg(p + 32 * k);
    }
    __device__ __forceinline__ int row() const { return (int)c[META].w; }
    __device__ __forceinline__ int own() const { return (int)(c[META].z & 0xffffu); }
    __device__ __forceinline__ int kp() const { return (int)((c[META].z >> 16) & 0xffu); }
    __device__ __forceinline__ bool write() const { return (c[META].z >> 24) != 0; }
    __device__ __forceinline__ int slot(int q) const
    {
        const unsigned w = q < 2 ? c[META].x : c[META].y;
        return (int)((q & 1) ? w >> 16 : w & 0xffffu);
    }
    __device__ __forceinline__ T v(int q) const;
    __device__ __forceinline__ T inv() const;
};
template <>
__device__ __forceinline__ double BandRec<double>::v(int q) const
{
    const uint4& p = c[q >> 1];
    return (q & 1) ? __hiloint2double((int)p.w, (int)p.z) : __hiloint2double((int)p.y, (int)p.x);
}
template <>
__device__ __forceinline__ double BandRec<double>::inv() const
{
    return __hiloint2double((int)c[3].y, (int)c[3].x);
}
template <>
__device__ __forceinline__ float BandRec<float>::v(int q) const
{
    return __uint_as_float(q == 0 ? c[0].x : q == 1 ? c[0].y : q == 2 ? c[0].z : c[0].w);
}
template <>
__device__ __forceinline__ float BandRec<float>::inv() const
{
    return __uint_as_float(c[2].x);
}

template <typename T, typename BT, int OUT>
__global__ void __launch_bounds__(32 * kBandWarps) k_sptrsv_band(const unsigned char* __restrict__ rec,
                                                                const int* __restrict__ ustep, int R,
                                                                const BT* __restrict__ b, T* x, double* x64)
{
    constexpr int rec_bytes = band_rec_bytes(sizeof(T));
    extern __shared__ __align__(16) unsigned char sm[];
    volatile T* ring = reinterpret_cast<volatile T*>(sm);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t0 = __ldg(ustep + blockIdx.x), ns = __ldg(ustep + blockIdx.x + 1) - t0;
    if (threadIdx.x == 0) ring[R] = (T)0;
    __syncthreads();
    BandRec<T> nxt, aft;  // the warp's next step and the one after
    T bn = (T)0;          // the next step's right-hand side
    auto rhs = [&](const BandRec<T>& z) -> T { return z.row() >= 0 ? (T)__ldg(b + z.row()) : (T)0; };
    if (warp < ns) {
        nxt.fetch(rec + (size_t)(t0 + warp) * rec_bytes, lane);
        bn = rhs(nxt);
    }
    if (warp + kBandWarps < ns) aft.fetch(rec + (size_t)(t0 + warp + kBandWarps) * rec_bytes, lane);
    for (int s = warp; s < ns; s += kBandWarps) {
        const BandRec<T> cur = nxt;
        const T bv = bn;
        if (s + kBandWarps < ns) {
            nxt = aft;
            bn = rhs(nxt);
        }
        if (s + 2 * kBandWarps < ns) aft.fetch(rec + (size_t)(t0 + s + 2 * kBandWarps) * rec_bytes, lane);
        const T v0 = -cur.v(0), v1 = -cur.v(1), v2 = -cur.v(2), v3 = -cur.v(3), inv = cur.inv();
        const int s0 = cur.slot(0), s1 = cur.slot(1), s2 = cur.slot(2), s3 = cur.slot(3);
        const int kp = cur.kp(), own = cur.own();
        const bool mine = own < R;
        if (s > 0) asm volatile("barrier.cta.sync %0, 64;" ::"r"(warp) : "memory");
        const T x0 = ring[s0], x1 = ring[s1], x2 = ring[s2], x3 = ring[s3];
        // two partial sums halve the dependent multiply-add chain
        T a0 = bv + v0 * x0, a1 = v1 * x1;
        a0 += v2 * x2;
        a1 += v3 * x3;
        T acc = a0 + a1;
        if (kp > 1) {
            if (kp > 2) {
                if (kp > 4) {
                    if (kp > 8) {
                        if (kp > 16) acc += __shfl_xor_sync(0xffffffffu, acc, 16);
                        acc += __shfl_xor_sync(0xffffffffu, acc, 8);
                    }
                    acc += __shfl_xor_sync(0xffffffffu, acc, 4);
                }
                acc += __shfl_xor_sync(0xffffffffu, acc, 2);
            }
            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        }
        const T xv = acc * inv;
        if (mine) ring[own] = xv;
        if (s + 1 < ns)
            asm volatile("barrier.cta.arrive %0, 64;" ::"r"((warp + 1) % kBandWarps) : "memory");
        if (cur.write()) {
            const int r = cur.row();
            if (x) x[r] = xv;
            if (OUT == OUT_SET64) x64[r] = (double)xv;
            if (OUT == OUT_ADD64) x64[r] += (double)xv;
        }
    }
}

template <typename T, typename BT, int OUT>
int band_launch_t(const BandLayout& t, const unsigned char* rec, const BT* b, T* x, double* x64, cudaStream_t s)
{
    auto kern = k_sptrsv_band<T, BT, OUT>;
    const size_t smem = (size_t)(t.R + 1) * sizeof(T);
    SPT_CUDA(allow_smem(kern, smem));
    kern<<<t.nunits, 32 * kBandWarps, smem, s>>>(rec, t.ustep, t.R, b, x, x64);
    SPT_CUDA(cudaGetLastError());
    return 0;
}

// f(0 .. n-1) over the host's threads; what a thread throws is thrown here,
// once all of them have ended.
template <class F>
void band_spread(int n, F&& f)
{
    const int nt = std::max(1, std::min<int>(n, (int)std::thread::hardware_concurrency()));
    std::vector<std::exception_ptr> err(nt);
    auto work = [&](int t) {
        try {
            for (int i = t; i < n; i += nt) f(i);
        } catch (...) {
            err[t] = std::current_exception();
        }
    };
    std::vector<std::thread> th;
    th.reserve(nt);
    int started = 1;  // threads 1 .. started - 1 run; their shares past those are done here
    try {
        for (; started < nt; started++) th.emplace_back(work, started);
    } catch (const std::system_error&) {
    }
    work(0);
    for (int t = started; t < nt; t++) work(t);
    for (auto& x : th) x.join();
    for (auto& e : err)
        if (e) std::rethrow_exception(e);
}

}  // namespace

void band_free(BandLayout& t)
{
    cudaFree(t.rec64); cudaFree(t.rec32); cudaFree(t.ustep); cudaFree(t.own_b);
    t = BandLayout{};
}

int download_natural_csr(sptrsv_plan_s* p, std::vector<int>& rp, std::vector<int>& ci, std::vector<double>& va);

int build_band_layout(sptrsv_plan_s* p)
{
    if (p->band.rec64) return 0;
    const int n = p->n, U = kBandU;
    std::vector<int> rp, ci;
    std::vector<double> va;
    int e = download_natural_csr(p, rp, ci, va);
    if (e) return e;
    std::vector<int> lev(n);
    if (n > 0) SPT_CUDA(cudaMemcpy(lev.data(), p->levels, sizeof(int) * (size_t)n, cudaMemcpyDeviceToHost));
    // units: the blocks of a block system, else the whole matrix
    std::vector<int> u0 = p->blk_starts;
    if (u0.empty()) u0.push_back(0);
    u0.push_back(n);
    const int nunits = (int)u0.size() - 1;
    // rows of the block system back to the outer plan's rows (partitioned plans)
    auto outer_row = [&](int unit, int r, bool* real) {
        if (p->part_tab.empty()) {
            *real = true;
            return r;
        }
        const int s = p->part_tab[4 * unit], a = p->part_tab[4 * unit + 1], base = p->part_tab[4 * unit + 3];
        const int o = s + (r - base);
        *real = o >= a;
        return o;
    };
    int maxoff = 0;
    for (int r = 0; r < n; r++) maxoff = std::max(maxoff, rp[r + 1] - rp[r] - 1);
    if (maxoff > 32 * U)
        return set_error(SPTRSV_ERR_UNSUPPORTED, "band schedule: a row holds %d off-diagonals, more than %d", maxoff,
                         32 * U);
    for (int un = 0; un < nunits; un++) {
        const int a = u0[un], b = u0[un + 1];
        int lmin = 1 << 30, lmax = 0;
        for (int r = a; r < b; r++) {
            lmin = std::min(lmin, lev[r]);
            lmax = std::max(lmax, lev[r]);
        }
        const int nl = b > a ? lmax - lmin + 1 : 0;
        if (b > a && (b - a) > 128 * nl)
            return set_error(SPTRSV_ERR_UNSUPPORTED, "band schedule: levels hold %d rows on average, too wide for one "
                             "CTA", (b - a) / nl);
    }
    // the units' steps and slots, the units spread over the host's threads
    std::vector<BandUnit> units(nunits);
    auto spread = [&](auto&& f) { band_spread(nunits, f); };
    spread([&](int un) {
        const int a = u0[un], b = u0[un + 1];
        band_unit(rp.data(), ci.data(), lev.data(), a, b, units[un]);
    });
    int R = 1;
    std::vector<int> ustep(nunits + 1, 0);
    for (int un = 0; un < nunits; un++) {
        R = std::max(R, units[un].R);
        ustep[un + 1] = ustep[un] + (int)units[un].steps.size();
    }
    if (R > kBandMaxRing)
        return set_error(SPTRSV_ERR_UNSUPPORTED, "band schedule: %d values are alive at once, more than the %d "
                         "shared-memory slots", R, kBandMaxRing);
    const long long ns = ustep[nunits];
    const int rb64 = band_rec_bytes(8), rb32 = band_rec_bytes(4);
    std::vector<unsigned char> h64((size_t)ns * rb64, 0), h32((size_t)ns * rb32, 0);
    spread([&](int un) {
        const BandUnit& u = units[un];
        const int a = u0[un];
        for (size_t t = 0; t < u.steps.size(); t++) {
            const BandStepHost& sp = u.steps[t];
            unsigned char* r64 = &h64[(ustep[un] + t) * rb64];
            unsigned char* r32 = &h32[(ustep[un] + t) * rb32];
            // per lane: values, slots (R: the constant-0 slot), row slot, outer row, 1/L_rr
            double v[32][4] = {};
            int sl[32][4], os[32], row[32], wr[32] = {};
            double inv[32] = {};
            float invf[32] = {};
            for (int j = 0; j < 32; j++) {
                for (int q = 0; q < 4; q++) sl[j][q] = R;
                os[j] = R;  // no row: slot R is never written
                row[j] = -1;
            }
            for (int w = 0; w < sp.cnt; w++) {
                const int r = u.order[sp.first + w];
                const int lane0 = w * sp.kp;
                const int d = rp[r + 1] - 1;
                for (int q = rp[r]; q < d; q++) {
                    const int k = q - rp[r];
                    const int lane = lane0 + (k % sp.kp), uu = k / sp.kp;
                    sl[lane][uu] = u.slot_of[ci[q] - a];
                    v[lane][uu] = va[q];
                }
                bool real = true;
                row[lane0] = outer_row(un, r, &real);
                wr[lane0] = real ? 1 : 0;
                os[lane0] = u.slot_of[r - a];
                inv[lane0] = 1.0 / va[d];
                invf[lane0] = 1.0f / (float)va[d];
            }
            for (int j = 0; j < 32; j++) {
                const unsigned meta[4] = {(unsigned)sl[j][0] | ((unsigned)sl[j][1] << 16),
                                          (unsigned)sl[j][2] | ((unsigned)sl[j][3] << 16),
                                          (unsigned)os[j] | ((unsigned)sp.kp << 16) | ((unsigned)wr[j] << 24),
                                          (unsigned)row[j]};
                // FP64 pieces
                memcpy(r64 + 0 * 512 + j * 16, &v[j][0], 16);
                memcpy(r64 + 1 * 512 + j * 16, &v[j][2], 16);
                memcpy(r64 + 2 * 512 + j * 16, meta, 16);
                memcpy(r64 + 3 * 512 + j * 16, &inv[j], 8);
                // FP32 pieces
                const float vf[4] = {(float)v[j][0], (float)v[j][1], (float)v[j][2], (float)v[j][3]};
                memcpy(r32 + 0 * 512 + j * 16, vf, 16);
                memcpy(r32 + 1 * 512 + j * 16, meta, 16);
                memcpy(r32 + 2 * 512 + j * 16, &invf[j], 4);
            }
        }
    });
    BandLayout t;
    t.U = U;
    t.R = R;
    t.nunits = nunits;
    t.nsteps = (int)ns;
    t.rb64 = rb64;
    t.rb32 = rb32;
    auto fail = [&](int code) {
        band_free(t);
        return code;
    };
    if (dalloc(&t.ustep, nunits + 1) != cudaSuccess || dalloc(&t.rec64, (long long)ns * rb64) != cudaSuccess ||
        dalloc(&t.rec32, (long long)ns * rb32) != cudaSuccess ||
        (!p->part_tab.empty() && dalloc(&t.own_b, p->part_tab[p->part_tab.size() - 2]) != cudaSuccess))
        return fail(cuda_fail(cudaGetLastError(), "band layout"));
    if (cudaMemcpy(t.ustep, ustep.data(), sizeof(int) * (size_t)(nunits + 1), cudaMemcpyHostToDevice) != cudaSuccess ||
        (ns > 0 && (cudaMemcpy(t.rec64, h64.data(), h64.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
                    cudaMemcpy(t.rec32, h32.data(), h32.size(), cudaMemcpyHostToDevice) != cudaSuccess)))
        return fail(cuda_fail(cudaGetLastError(), "band layout upload"));
    p->band = t;
    return 0;
}

// One BAND solve: b (FP64 or FP32, in the outer plan's rows), one CTA per unit.
// x (T) and x64 per out_mode; x may be null.
int band_solve(sptrsv_plan_s* p, bool f32, const void* b, bool b_f32, void* x, double* x64, int out_mode,
               cudaStream_t s)
{
    int e = build_band_layout(p);
    if (e) return e;
    const BandLayout& t = p->band;
    if (t.nsteps == 0) return 0;
    const double* bd = static_cast<const double*>(b);
    const float* bf = static_cast<const float*>(b);
    if (t.own_b) {
        // warm-up rows read b of rows that another unit writes the result of: a solve in place takes a copy of b
        const size_t m = (size_t)p->part_tab[p->part_tab.size() - 2];  // end of the last block
        const size_t bytes = m * (b_f32 ? sizeof(float) : sizeof(double));
        auto overlaps = [&](const void* y, size_t elem) {
            return y && (uintptr_t)y < (uintptr_t)b + bytes && (uintptr_t)b < (uintptr_t)y + m * elem;
        };
        if (overlaps(x, f32 ? sizeof(float) : sizeof(double)) || overlaps(x64, sizeof(double))) {
            SPT_CUDA(cudaMemcpyAsync(t.own_b, b, bytes, cudaMemcpyDeviceToDevice, s));
            bd = t.own_b;
            bf = reinterpret_cast<const float*>(t.own_b);
        }
    }
    if (!f32) return band_launch_t<double, double, OUT_X>(t, t.rec64, bd, static_cast<double*>(x), nullptr, s);
    float* xf = static_cast<float*>(x);
    if (out_mode == OUT_SET64)
        return b_f32 ? band_launch_t<float, float, OUT_SET64>(t, t.rec32, bf, xf, x64, s)
                     : band_launch_t<float, double, OUT_SET64>(t, t.rec32, bd, xf, x64, s);
    if (out_mode == OUT_ADD64)
        return b_f32 ? band_launch_t<float, float, OUT_ADD64>(t, t.rec32, bf, xf, x64, s)
                     : band_launch_t<float, double, OUT_ADD64>(t, t.rec32, bd, xf, x64, s);
    return b_f32 ? band_launch_t<float, float, OUT_X>(t, t.rec32, bf, xf, x64, s)
                 : band_launch_t<float, double, OUT_X>(t, t.rec32, bd, xf, x64, s);
}

}  // namespace sptrsv
