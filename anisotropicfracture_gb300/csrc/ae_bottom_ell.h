// The assembled coarsest-level matrix in the layout of the four-warp bottom solve (host code).
#pragma once
#include <algorithm>
#include <numeric>
#include <vector>

namespace ae {

constexpr int kEllWarps = 4, kEllThreads = 32 * kEllWarps;
constexpr int kEllLongRow = 4;  // rows of more chunks are summed by 8 lanes

// Unknowns sit in slots: thread t of 128 holds slots t, t + 128, ...  perm[slot] = unknown (-1: none);
// rows[slot] = first chunk | number of chunks << 16 (0: none).  A row is cut into chunks of at most
// `chunk` nonzeros; the chunks, longest first, fill groups of 32, and warp w runs the groups
// [wgrp[w], wgrp[w + 1]).  Step q of group g multiplies val[goff[g] + 32 q + lane] by the vector
// entry (slot) col[...] for the lanes whose chunk is longer than q; slot[32 g + lane] = chunk |
// (length + 1) << 16 (0: no chunk).  A row of more than kEllLongRow chunks sits on a lane that is a
// multiple of 8, so that it and the next 7 lanes can add its chunks' sums together.
struct BottomEllHost {
    std::vector<double> val;
    std::vector<unsigned short> col;
    std::vector<int> goff, slot, wgrp, rows, perm;
    int nchunk = 0, layers = 0, chunk = 0;
    bool ok = false;
};

// warp-wide FP64 instructions of one product on the busiest warp, for chunks of c nonzeros
inline int bottom_ell_cost(const std::vector<int>& lens, int c) {
    std::vector<int> count(c + 1, 0);  // chunks of each length
    int most = 1;
    for (int n : lens) {
        most = std::max(most, (n + c - 1) / c);
        count[c] += n / c;
        count[n % c] += 1;
    }
    // groups of 32 chunks, longest first: each as long as its first
    int load[kEllWarps] = {};
    int len = c, before = 0;  // chunks longer than len
    for (int g = 0;; g += 32) {
        while (len > 0 && g >= before + count[len]) before += count[len--];
        if (len == 0) break;
        *std::min_element(load, load + kEllWarps) += len;
    }
    return *std::max_element(load, load + kEllWarps) + (most > kEllLongRow ? 3 + (most - 1) / 8 : most - 1);
}

inline BottomEllHost bottom_ell(const std::vector<int>& rowptr, const std::vector<int>& col,
                                const std::vector<double>& val, int max_layers) {
    BottomEllHost h;
    const int N = (int)rowptr.size() - 1;
    if (N < 1 || N > max_layers * kEllThreads) return h;
    std::vector<int> lens(N), byrow(N);
    for (int r = 0; r < N; ++r) lens[r] = rowptr[r + 1] - rowptr[r];
    int best = 0;
    for (int c = 3; c <= 16; ++c) {
        const int cost = bottom_ell_cost(lens, c);
        if (!h.chunk || cost < best) h.chunk = c, best = cost;
    }
    // slots: the long rows, longest first, on every eighth lane; the others in the gaps
    std::iota(byrow.begin(), byrow.end(), 0);
    std::stable_sort(byrow.begin(), byrow.end(), [&](int a, int b) { return lens[a] > lens[b]; });
    std::vector<int> slot_of(N, -1);
    int nlong = 0;
    while (nlong < N && lens[byrow[nlong]] > kEllLongRow * h.chunk) {
        slot_of[byrow[nlong]] = 8 * nlong;
        ++nlong;
    }
    int top = nlong ? 8 * (nlong - 1) + 1 : 0;
    for (int n = nlong, at = 0; n < N; ++n, ++at) {
        while (at % 8 == 0 && at / 8 < nlong) ++at;
        slot_of[byrow[n]] = at;
        top = std::max(top, at + 1);
    }
    h.layers = (top + kEllThreads - 1) / kEllThreads;
    if (h.layers > max_layers) return h;
    h.perm.assign((size_t)h.layers * kEllThreads, -1);
    h.rows.assign(h.perm.size(), 0);
    std::vector<int> begin, count;  // per chunk: first nonzero (of the CSR arrays) and length
    for (int r = 0; r < N; ++r) {
        const int first = (int)begin.size();
        int q = rowptr[r];
        do {
            const int e = std::min(q + h.chunk, rowptr[r + 1]);
            begin.push_back(q);
            count.push_back(e - q);
            q = e;
        } while (q < rowptr[r + 1]);
        h.perm[slot_of[r]] = r;
        h.rows[slot_of[r]] = first | ((int)begin.size() - first) << 16;
    }
    h.nchunk = (int)begin.size();
    if (h.nchunk > 65535) return h;
    std::vector<int> order(h.nchunk);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return count[a] > count[b]; });
    // groups to warps: each to the warp with the fewest steps so far
    std::vector<std::vector<int>> mine(kEllWarps);
    int load[kEllWarps] = {};
    for (int g = 0; 32 * g < h.nchunk; ++g) {
        const int w = (int)(std::min_element(load, load + kEllWarps) - load);
        load[w] += count[order[32 * g]];
        mine[w].push_back(g);
    }
    h.goff.push_back(0);
    h.wgrp.push_back(0);
    for (int w = 0; w < kEllWarps; ++w) {
        for (int g : mine[w]) {
            const int base = h.goff.back(), width = count[order[32 * g]];
            h.val.resize((size_t)base + 32 * width, 0.0);
            h.col.resize((size_t)base + 32 * width, 0);
            for (int l = 0; l < 32; ++l) {
                if (32 * g + l >= h.nchunk) {
                    h.slot.push_back(0);
                    continue;
                }
                const int c = order[32 * g + l];
                for (int q = 0; q < count[c]; ++q) {
                    h.val[base + 32 * q + l] = val[begin[c] + q];
                    h.col[base + 32 * q + l] = (unsigned short)slot_of[col[begin[c] + q]];
                }
                h.slot.push_back(c | (count[c] + 1) << 16);
            }
            h.goff.push_back(base + 32 * width);
        }
        h.wgrp.push_back((int)h.goff.size() - 1);
    }
    h.ok = true;
    return h;
}

}  // namespace ae
