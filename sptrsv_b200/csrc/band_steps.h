// band_steps.h — the BAND schedule's steps and slots, on the host (band.cu).
#pragma once

#include <algorithm>
#include <utility>
#include <vector>

namespace sptrsv {

constexpr int kBandU = 4;           // entries per lane per step
constexpr int kBandMaxRing = 8192;  // shared-memory slots

// One step: rows [first, first + cnt) of the unit's step order, kp lanes each.
struct BandStepHost {
    int kp, first, cnt;
};

// The steps of one unit: rows [a, b) of the natural CSR, all of whose columns
// lie in it, with their levels.
struct BandUnit {
    std::vector<BandStepHost> steps;
    std::vector<int> order;    // rows in step order
    std::vector<int> slot_of;  // by row - a
    int R = 1;
};

inline int band_lanes(int len)
{
    int kp = 1;
    while ((len + kp - 1) / kp > kBandU) kp *= 2;
    return kp;
}

// List scheduling: of the rows whose columns lie in earlier steps, those with
// the longest chain of readers first; the first one's lane count is the
// step's, rows that need more wait.  Ready rows stand in one heap per lane
// count, longest chain first and among equals the one that came last, so a
// step looks at no row that it does not take: n = 400,000 in a band of 16 in
// 0.1 s, where a walk over all chain lengths a step took 33 s.
inline void band_list_steps(const int* rp, const int* ci, int a, int b, BandUnit& u)
{
    const int n = b - a;
    std::vector<int> height(n, 0), missing(n), cptr(n + 1, 0);
    for (int r = b - 1; r >= a; r--) {
        missing[r - a] = rp[r + 1] - 1 - rp[r];
        for (int q = rp[r]; q < rp[r + 1] - 1; q++) {
            int& h = height[ci[q] - a];
            h = std::max(h, height[r - a] + 1);
            cptr[ci[q] - a + 1]++;
        }
    }
    for (int i = 0; i < n; i++) cptr[i + 1] += cptr[i];
    std::vector<int> reader(cptr[n]), at(cptr.begin(), cptr.end() - 1);
    for (int r = a; r < b; r++)
        for (int q = rp[r]; q < rp[r + 1] - 1; q++) reader[at[ci[q] - a]++] = r;
    struct Ready {
        int height, came, row;
        bool operator<(const Ready& o) const { return height != o.height ? height < o.height : came < o.came; }
    };
    std::vector<Ready> heap[6];  // rows of 1 << j lanes
    int came = 0;
    auto add = [&](int r) {
        int j = 0;
        while ((1 << j) < band_lanes(rp[r + 1] - 1 - rp[r])) j++;
        heap[j].push_back({height[r - a], came++, r});
        std::push_heap(heap[j].begin(), heap[j].end());
    };
    for (int r = b - 1; r >= a; r--)
        if (missing[r - a] == 0) add(r);
    u.steps.clear();
    u.order.clear();
    u.order.reserve(n);
    while ((int)u.order.size() < n) {
        const int first = (int)u.order.size();
        int top = 5, per = 1;  // rows of up to 1 << top lanes; the first row takes any
        for (int k = 0; k < per; k++) {
            int best = -1;
            for (int j = 0; j <= top; j++)
                if (!heap[j].empty() && (best < 0 || heap[best][0] < heap[j][0])) best = j;
            if (best < 0) break;
            if (k == 0) {
                top = best;
                per = 32 >> best;
            }
            u.order.push_back(heap[best][0].row);
            std::pop_heap(heap[best].begin(), heap[best].end());
            heap[best].pop_back();
        }
        const int cnt = (int)u.order.size() - first;
        u.steps.push_back({1 << top, first, cnt});
        for (int k = first; k < first + cnt; k++) {
            const int i = u.order[k] - a;
            for (int q = cptr[i]; q < cptr[i + 1]; q++)
                if (--missing[reader[q] - a] == 0) add(reader[q]);
        }
    }
}

// Steps along the levels: every level cut by itself, its lane count from its
// longest row.
inline void band_level_steps(const int* rp, const int* lev, int a, int b, BandUnit& u)
{
    u.steps.clear();
    u.order.resize(b - a);
    for (int r = a; r < b; r++) u.order[r - a] = r;
    std::stable_sort(u.order.begin(), u.order.end(), [&](int p, int q) { return lev[p] < lev[q]; });
    for (int f = 0; f < b - a;) {
        int e = f, mx = 0;
        for (; e < b - a && lev[u.order[e]] == lev[u.order[f]]; e++)
            mx = std::max(mx, rp[u.order[e] + 1] - 1 - rp[u.order[e]]);
        const int kp = band_lanes(mx), per = 32 / kp;
        for (int q = f; q < e; q += per) u.steps.push_back({kp, q, std::min(per, e - q)});
        f = e;
    }
}

// Slots by interval allocation over the steps; false when more than
// kBandMaxRing values are alive at once.
inline bool band_slots(const int* rp, const int* ci, int a, int b, BandUnit& u)
{
    const int n = b - a, ns = (int)u.steps.size();
    std::vector<int> last(n, -1), step(n);
    for (int t = 0; t < ns; t++)
        for (int k = u.steps[t].first; k < u.steps[t].first + u.steps[t].cnt; k++) {
            const int r = u.order[k];
            step[r - a] = t;
            for (int q = rp[r]; q < rp[r + 1] - 1; q++) last[ci[q] - a] = t;  // steps ascend
        }
    std::vector<int> rptr(ns + 1, 0);
    for (int i = 0; i < n; i++) rptr[std::max(last[i], step[i]) + 1]++;
    for (int t = 0; t < ns; t++) rptr[t + 1] += rptr[t];
    std::vector<int> rel(n), at(rptr.begin(), rptr.end() - 1), freel;
    u.slot_of.assign(n, 0);
    int top = 0;
    for (int t = 0; t < ns; t++) {
        for (int k = u.steps[t].first; k < u.steps[t].first + u.steps[t].cnt; k++) {
            const int i = u.order[k] - a;
            int sl;
            if (!freel.empty()) {
                sl = freel.back();
                freel.pop_back();
            } else {
                sl = top++;
            }
            u.slot_of[i] = sl;
            rel[at[std::max(last[i], t)]++] = sl;
        }
        for (int k = rptr[t]; k < rptr[t + 1]; k++) freel.push_back(rel[k]);  // free from the next step on
    }
    u.R = std::max(1, top);
    return u.R <= kBandMaxRing;
}

// The unit's steps and slots: the shorter of the two cuts among those whose
// values fit the slots (narrow levels: a list of mixed lane counts can be the
// longer one, 137,458 against 127,081 steps for n = 400,000 in a band of 16).
inline void band_unit(const int* rp, const int* ci, const int* lev, int a, int b, BandUnit& u)
{
    band_list_steps(rp, ci, a, b, u);
    const bool fits = band_slots(rp, ci, a, b, u);
    BandUnit l;
    band_level_steps(rp, lev, a, b, l);
    if (fits && u.steps.size() <= l.steps.size()) return;
    if (band_slots(rp, ci, a, b, l) || !fits) u = std::move(l);
}

}  // namespace sptrsv
