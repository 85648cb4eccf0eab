// The launch rules of the split sweeps (csrc/ae_split_rules.h): a chunking of planes covers them, is not finer
// than three planes, and is none of those measured well behind the best; the sizes taken keep every offset an
// int.  Exit status 0 when every case holds.
#include <cstdio>
#include <initializer_list>

#include "ae_split_rules.h"

int main() {
    for (int nz = 1; nz <= 300; ++nz)
        for (long long tiles : {1ll, 2ll, 9ll, 30ll, 64ll, 85ll, 126ll, 152ll, 153ll, 256ll, 1000ll, 12321ll}) {
            const int kz = ae::tile_kz(tiles, nz, 152);
            if (kz < 1 || kz > nz || (nz >= 3 && kz < 3)) {
                std::printf("tiles %lld, %d planes: chunks of %d\n", tiles, nz, kz);
                return 1;
            }
        }
    // tiles, planes, and the chunk sizes measured within 6 % of the best of twelve (9 slots, product)
    const struct {
        int tiles, nz, good[10];
    } cases[] = {
        {56, 111, {23, 14, 13}},         {60, 119, {24}},
        {64, 127, {32, 19, 15, 11}},     {85, 135, {27, 20, 14}},
        {90, 143, {29}},                 {95, 151, {51, 26, 19, 16}},
        {126, 167, {28, 24, 21, 19}},    {132, 175, {88, 59, 44, 35, 30, 25, 22, 20, 18, 15}},
        {144, 191, {96, 64, 48, 39, 32, 28, 24, 22, 20}},
    };
    for (const auto& c : cases) {
        const int kz = ae::tile_kz(c.tiles, c.nz, 152);
        bool ok = false;
        for (int g : c.good) ok = ok || g == kz;
        if (!ok) {
            std::printf("tiles %d, %d planes: chunks of %d\n", c.tiles, c.nz, kz);
            return 1;
        }
    }
    // cubes of n nodes an edge, rows padded to 4: taken as long as the last offset a tile can form, two planes
    // past the box and a tile's columns and rows past the last plane, is an int
    for (long long n = 17; n < 1400; ++n) {
        const long long px = (n + 3) / 4 * 4, sz = px * n, sc = sz * n, last = sz * (n + 2) + px * 8 + 32;
        if (ae::split_range(sz, sc) ? last > 2147483647ll : n <= 1200) {
            std::printf("%lld nodes an edge\n", n);
            return 1;
        }
    }
    std::printf("ok\n");
    return 0;
}
