// Launch rules of the split sweeps (host code).
#pragma once

namespace ae {

// Planes per block of the FP64 tiled kernel: the split of nz planes into chunks that takes the fewest plane
// times.  wave: the blocks that run at once; a block goes through its own planes, two more and about one
// plane's time until its first plane has arrived.  A single wave counts a fifth more: nothing evens its
// blocks out (they differ in the nodes at grain boundaries and in the columns of edge tiles), while from two
// waves on an SM that is done early takes the next block.  Interior products in FP64, us, chunk sizes 64 / 19
// planes of 127 at 64 tiles: 9 slots 267 / 219, 21 slots 644 / 537; counting six planes a block and no more
// for a single wave took the first.
inline int tile_kz(long long tiles, int nz, long long wave) {
    int best = nz;
    long long cost = -1;
    for (int n = 1; n <= (nz + 3) / 4; ++n) {
        const int kz = (nz + n - 1) / n;
        const long long waves = (tiles * ((nz + kz - 1) / kz) + wave - 1) / wave;
        const long long c = waves * (kz + 3) * (waves == 1 ? 12 : 10);
        if (cost < 0 || c < cost) cost = c, best = kz;
    }
    return best;
}

// Whether the tiled kernels can index an array of planes of sz elements, sc elements a component: offsets
// inside a component are 32-bit (the components' own are not), and run a few planes past the box.  897^3 nodes,
// two slots, FP64 product: 90.4 ms, per node 134.6, the same bits.
inline bool split_range(long long sz, long long sc) { return sc + 8 * sz < (1ll << 31); }

}  // namespace ae
