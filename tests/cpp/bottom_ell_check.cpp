// bottom_ell (the four-warp bottom solve's matrix layout) on random sparse matrices: its product,
// formed group by group as the kernel does, equals the CSR product.  Exit status 0 when it holds.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "ae_bottom_ell.h"

int main() {
    std::mt19937 rng(3);
    const auto uni = [&] { return (double)rng() / 4.3e9 - 0.5; };
    for (int trial = 0; trial < 300; ++trial) {
        const int N = 1 + (int)(rng() % 600);
        std::vector<int> rp(1, 0), col;
        std::vector<double> val;
        for (int i = 0; i < N; ++i) {  // empty rows among them
            const int len = (int)(rng() % 4 ? rng() % 3 : rng() % 65);
            for (int q = 0; q < len; ++q) {
                col.push_back((int)(rng() % N));
                val.push_back(uni());
            }
            rp.push_back((int)col.size());
        }
        const ae::BottomEllHost h = ae::bottom_ell(rp, col, val, 64);
        if (!h.ok || h.perm.size() != (size_t)h.layers * ae::kEllThreads || h.wgrp.size() != ae::kEllWarps + 1) return 1;
        if (h.slot.size() != 32 * (h.goff.size() - 1) || h.wgrp.back() + 1 != (int)h.goff.size()) return 1;
        std::vector<double> x(N), xs(h.perm.size(), 0.0), part(h.nchunk, 1e300);
        std::vector<int> seen(N, 0);
        for (double& v : x) v = uni();
        for (size_t n = 0; n < h.perm.size(); ++n)
            if (h.perm[n] >= 0) {
                xs[n] = x[h.perm[n]];
                ++seen[h.perm[n]];
            }
        for (int v : seen)
            if (v != 1) return 2;
        for (int w = 0; w < ae::kEllWarps; ++w)
            for (int g = h.wgrp[w]; g < h.wgrp[w + 1]; ++g)
                for (int l = 0; l < 32; ++l) {
                    const int t = h.slot[32 * g + l], len = (t >> 16) - 1;
                    if (!t) continue;
                    if (len > h.chunk || 32 * len > h.goff[g + 1] - h.goff[g]) return 3;
                    double s = 0.0;
                    for (int q = 0; q < len; ++q) s += h.val[h.goff[g] + 32 * q + l] * xs[h.col[h.goff[g] + 32 * q + l]];
                    part[t & 0xffff] = s;
                }
        for (size_t n = 0; n < h.perm.size(); ++n) {
            const int first = h.rows[n] & 0xffff, cnt = h.rows[n] >> 16, r = h.perm[n];
            if ((r < 0) != (cnt == 0) || (cnt > ae::kEllLongRow && n % 8)) return 4;
            if (r < 0) continue;
            double s = 0.0, ref = 0.0;
            for (int c = 0; c < cnt; ++c) s += part[first + c];
            for (int q = rp[r]; q < rp[r + 1]; ++q) ref += val[q] * x[col[q]];
            if (!(std::fabs(s - ref) < 1e-13)) {
                std::printf("trial %d row %d: %g, not %g\n", trial, r, s, ref);
                return 5;
            }
        }
    }
    return 0;
}
