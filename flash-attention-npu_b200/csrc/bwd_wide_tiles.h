// Which 128-row blocks of a sequence meet in the backward above head dim 128, and where their stored tiles lie.  Plain C++:
// the kernels of bwd_wide_sm100.cu and a CPU test of the index range compile the same lines.
#pragma once
#include <cstddef>

#ifdef __CUDACC__
#define FA_HD __host__ __device__ __forceinline__
#else
#define FA_HD inline
#endif

namespace fa {

constexpr size_t kWideTileBytes = 128 * 128 * 2;             // one stored P^T or dS^T tile

// Blocks of the tile grid of a head: the workspace holds nkb x nqb tiles, from the longest lengths that the caller names.
// A packed sequence that is longer than it said keeps to the grid (its gradients are then incomplete, as its query rows
// past the stated length are with the other kernels), so that no tile lies outside the workspace.
struct WideGrid {
    int nkb, nqb;
    int causal, wl, wr;
};
struct BlockRange {
    int lo, hi;
};

// query blocks [lo, hi) that key block n of a sequence is visible to: the one rule both kernels go by
FA_HD BlockRange wide_query_blocks(const WideGrid& t, int sq, int sk, int n) {
    const int n0 = n * 128, krows = sk - n0 < 128 ? sk - n0 : 128, diff = sk - sq;
    const int wr = t.causal ? 0 : t.wr;
    int i_lo = 0, i_hi = sq - 1;
    if (wr >= 0 && n0 - diff - wr > 0) i_lo = n0 - diff - wr;
    if (t.wl >= 0 && n0 + krows - 1 + t.wl - diff < i_hi) i_hi = n0 + krows - 1 + t.wl - diff;
    BlockRange r;
    r.lo = i_lo / 128 < t.nqb ? i_lo / 128 : t.nqb;
    r.hi = r.lo;
    if (n < t.nkb && n0 < sk && i_hi >= i_lo) r.hi = i_hi / 128 + 1 < t.nqb ? i_hi / 128 + 1 : t.nqb;
    return r;
}

// key blocks that reach query block m: the n for which wide_query_blocks holds m, one range
FA_HD BlockRange wide_key_blocks(const WideGrid& t, int sq, int sk, int m) {
    const int diff = sk - sq, wr = t.causal ? 0 : t.wr;
    const int blocks = (sk + 127) / 128 < t.nkb ? (sk + 127) / 128 : t.nkb;
    const int last = m * 128 + 127 < sq - 1 ? m * 128 + 127 : sq - 1;                // last row of the block
    BlockRange r;
    r.lo = 0;
    r.hi = m < t.nqb && m * 128 < sq ? blocks : 0;
    if (wr >= 0) {                                           // the block's first key is at most wr past some row's diagonal
        const int key = last + diff + wr;
        const int hi = key < 0 ? 0 : key / 128 + 1;
        if (hi < r.hi) r.hi = hi;
    }
    if (t.wl >= 0) {                                         // the block's last key is at most wl before the first row's diagonal
        const int key = m * 128 + diff - t.wl;
        if (key > sk - 1) r.hi = 0;
        else if (key > 0) r.lo = key / 128;
    }
    return r;
}

// byte offset of tile (pair of the launch, head of the group, key block, query block)
FA_HD size_t wide_tile_at(const WideGrid& t, int group, int pair, int g, int n, int m) {
    return ((((size_t)pair * group + g) * t.nkb + n) * t.nqb + m) * kWideTileBytes;
}

}  // namespace fa
