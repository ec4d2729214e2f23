// Host side of block.cuh: which states of a system couple to the detection
// states, and how their rows are laid out on the lanes of a CTA.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <numeric>
#include <vector>

namespace spx {

// Connected components of a symmetric pattern: label[i] of every row.
struct Components {
    std::vector<int> parent;
    explicit Components(int n) : parent(n) { std::iota(parent.begin(), parent.end(), 0); }
    int find(int i) {
        while (parent[i] != i) i = parent[i] = parent[parent[i]];
        return i;
    }
    void join(int a, int b) {
        a = find(a);
        b = find(b);
        if (a != b) parent[std::max(a, b)] = std::min(a, b);
    }
};

// The coupled rows and everything a layout needs, in numbers of their own
// (0 .. n-1, in the order of the system's rows).
struct BlockPattern {
    struct Entry { int col, src; };           // as BlockLayout::col and src
    int n = 0, nv = 0;
    std::vector<int> rows;                    // system row of every coupled row
    std::vector<std::vector<Entry>> entries;  // n state rows, then nv detection rows
    std::vector<double> values;               // detection rows' values
    std::vector<int> vchan, vfac;
};

// One assignment of the rows to the lanes of a CTA of 32 * warps threads.  A
// row takes a power of two of neighbouring lanes (its parts), each with at
// most `entries` of its entries; rows go to the lanes in decreasing order of
// parts, so the groups stay aligned, and of entries, so that the lanes of a
// warp end their loops together.
struct BlockLanes {
    int warps = 0, ecap = 0;
    std::vector<int> row, part, shape, src;   // see BlockLayout
    std::vector<uint16_t> col;
};

// Cost model of a term (cycles): what its warps issue, and how long it takes end
// to end (the busiest of the SM's four units, warp w on unit w mod 4).  FP32
// (measured on GB300): an entry is five packed multiply-adds of two FMA cycles
// and a load, a split row's reduction step about 55 cycles, the rest of a term
// 45 to issue and about 120 of latency.  FP64: one instruction holds a warp and its FP64
// unit for 64 cycles and the SM has four units; a row is two lanes (real and
// imaginary part), each with one instruction per entry and reduction step and
// three or four of its own.
struct BlockCost {
    double issue = 0.0;        // all warps of one orientation, cycles of the SM's unit
    double latency = 0.0;
    int warps = 0;             // of one orientation's CTA
    int warps_per_sm = 16;     // resident, by registers
    // a Lanczos step of the FP64 bounds on this layout, alike: one instruction (two
    // with complex couplings) per entry and reduction step, and about 30 of its own
    double bounds_issue = 0.0, bounds_latency = 0.0;
    int bounds_warps = 0;
    double bounds_time(double per_sm) const {
        const double res = std::max(1.0, std::floor(16.0 / bounds_warps)), full = std::floor(per_sm / res);
        const double rest = std::ceil(per_sm - full * res);
        return full * std::max(bounds_latency, res * bounds_issue) +
               (rest > 0.0 ? std::max(bounds_latency, rest * bounds_issue) : 0.0);
    }
    // relative time of n orientations per SM: rounds of as many as fit, the last
    // with what is left
    double time(double per_sm) const {
        const double res = std::max(1.0, std::floor((double)warps_per_sm / warps)), full = std::floor(per_sm / res);
        const double rest = std::ceil(per_sm - full * res);
        return full * std::max(latency, res * issue) + (rest > 0.0 ? std::max(latency, rest * issue) : 0.0);
    }
};

inline int pow2_ceil(int x) {
    int p = 1;
    while (p < x) p *= 2;
    return p;
}

// Lanes that the rows take with at most e entries each.
inline size_t block_lane_count(const BlockPattern &P, int e) {
    size_t lanes = 0;
    for (auto &r : P.entries) {
        const int parts = pow2_ceil(((int)r.size() + e - 1) / e);
        if (parts > 32) return (size_t)1 << 30;
        lanes += parts;
    }
    return lanes;
}

// The layout on `warps` warps with at most e entries per lane; false if the
// rows do not fit.
inline bool block_lanes(const BlockPattern &P, int warps, int e, bool f64, bool damped, bool cplx, BlockLanes &L,
                        BlockCost &cost) {
    if (block_lane_count(P, e) > 32u * (size_t)warps) return false;
    const int T = 32 * warps, nr = P.n + P.nv;
    std::vector<int> parts(nr), per(nr), order(nr);
    for (int r = 0; r < nr; ++r) {
        const int w = (int)P.entries[r].size();
        parts[r] = pow2_ceil((w + e - 1) / e);
        per[r] = (w + parts[r] - 1) / parts[r];
        order[r] = r;
    }
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        return parts[a] != parts[b] ? parts[a] > parts[b] : per[a] > per[b];
    });
    L.warps = warps;
    L.ecap = e;
    L.row.assign(T, -1);
    L.part.assign(T, 1);
    L.shape.assign(warps, 0);
    L.src.assign((size_t)e * T, -1);
    L.col.assign((size_t)e * T, 0);
    std::vector<int> ew(warps, 0), rounds(warps, 0);
    int t = 0;
    for (int r : order) {
        for (int q = 0; q < parts[r]; ++q, ++t) {
            L.row[t] = r;
            L.part[t] = parts[r] | (q << 8);
            const int w0 = q * per[r], w1 = std::min<int>((int)P.entries[r].size(), w0 + per[r]);
            for (int i = w0; i < w1; ++i) {
                L.src[(size_t)(i - w0) * T + t] = P.entries[r][i].src;
                L.col[(size_t)(i - w0) * T + t] = (uint16_t)P.entries[r][i].col;
            }
            ew[t / 32] = std::max(ew[t / 32], per[r]);
            int lg = 0;
            while ((1 << lg) < parts[r]) ++lg;
            rounds[t / 32] = std::max(rounds[t / 32], lg);
        }
    }
    cost = BlockCost{};
    cost.warps = f64 ? 2 * warps : warps;
    cost.warps_per_sm = f64 ? 32 : 16;
    double unit[4] = {0.0, 0.0, 0.0, 0.0}, bunit[4] = {0.0, 0.0, 0.0, 0.0};
    cost.bounds_warps = warps;
    for (int w = 0; w < warps; ++w) {
        L.shape[w] = ew[w] | (rounds[w] << 8);
        const double b = 64.0 * ((cplx ? 2.0 : 1.0) * (ew[w] + rounds[w]) + 30.0);
        cost.bounds_issue += b / 4.0;
        bunit[w % 4] += b;
        if (f64) {
            const double n = 64.0 * (ew[w] + rounds[w] + (damped ? 4.0 : 3.0));
            cost.issue += 2.0 * n / 4.0;
            unit[w % 4] += n;
            unit[(w + warps) % 4] += n;
            cost.latency = std::max(cost.latency, n);
        } else {
            // code instances (block_dispatch): entries in steps, the whole with split rows
            const int cap = e <= 4 ? 4 : e <= 8 ? 8 : (e + 7) / 8 * 8;
            const int step = cap <= 8 ? 1 : cap / 8;
            const double n = rounds[w] ? cap : std::max(step, (ew[w] + step - 1) / step * step);
            const double r = rounds[w] > 2 ? 5 : rounds[w];
            const double own = 11.0 * n + 20.0 * r + 45.0;
            cost.issue += own / 4.0;
            unit[w % 4] += own;
            cost.latency = std::max(cost.latency, own + 35.0 * r);
        }
    }
    for (double u : unit) cost.latency = std::max(cost.latency, u);
    for (double u : bunit) cost.bounds_latency = std::max(cost.bounds_latency, u);
    cost.latency += f64 ? 200.0 : 120.0;
    if (cost.warps > 1) cost.latency += 30.0;
    return true;
}

}  // namespace spx
