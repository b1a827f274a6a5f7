// When the last level runs as micro-ops (leaf_level_kernel) and when word by
// word (point_level_kernel). Both build the same masks. Plain C++ for both sides:
// the host leaves the first out of launches where it would not be picked, the
// level scan picks.
#pragma once
#include <cstdint>

#if defined(__CUDACC__)
#define FREP_LR_HD __host__ __device__ __forceinline__
#else
#define FREP_LR_HD inline
#endif

namespace frep {

// The fewest cells of a launch's last level for which leaf_pays picks the pass
// over micro-ops, but for few nodes with long tapes: of nodes of dim 4 and of
// larger ones.
constexpr unsigned long long kLeafCells4 = 7ull << 20, kLeafCells8 = 3ull << 20;

// Whether a tree's last level is worth the pass over micro-ops: nodes of dim^3
// cells and of `words` words on average, of a root tape with `root` words
// (transcendental: with a SIN, COS or EXP), in a launch of `cells` cells. Decoding pays once a warp has enough to share and to overlap, so the line
// is a number of cells, and it lies higher the less a tape loses by decoding. Word
// by word and as micro-ops, ms:
//   * 40 to 150 words, dim 4: 2 M cells .073 .093, 12 M .85 .85, 49 M 3.05 1.95;
//     dim 8: 3.9 M .14 .16, 14 M .39 .33, 110 M 2.3 1.4
//   * 16 words: 9 M .11 .12, 36 M .37 .26
//   * whole tapes of 19 and 26 words (no operation folds): dim 4 37 M .64 .60, 183
//     M 1.93 1.27; dim 8 never (366 M 2.39 2.45)
//   * sine and cosine, most of the time of such a tape in either pass: dim 4 with
//     46 words never (99 M 2.53 2.63, 245 M 11.1 12.1), with 239 words 140 M 7.3
//     6.6; dim 8 2 M .13 .13, 6.9 M .36 .26, 50 M 2.75 1.23
//   * 200 words and more, dim 8: 4.8 M .38 .33, but a warp needs about twenty items
//     per hundred words against the tail (6.3 M of 1,681 words 2.9 4.2)
//   (Scenes differ: where most leaf tapes need more than 14 rows and so run 2 cells
//   per lane, as in 2 of 23 scenes of 14 to 40 primitives, words stay 10 to 25 %
//   faster at any size, and nothing known before the pass tells them apart.)
//   * up to 2,048 nodes of dim 4 (a warp has one): 850 words .29 .24, 80 words .052
//     .048, 44 words .028 .030
FREP_LR_HD bool leaf_pays(uint32_t dim, bool transcendental, unsigned long long root, unsigned long long words,
                          unsigned long long cells) {
    const bool small = dim == 4;
    if (small && cells <= 1ull << 17) return words >= 80;
    if (root < 32) return small && cells >= 1ull << 25;
    if (transcendental) return small ? root >= 128 && cells >= 1ull << 26 : cells >= kLeafCells8;
    if (words < 18) return cells >= 1ull << 25;
    if (words >= 200 && !small) return cells >= kLeafCells8 && cells >= 22ull * 256 * words;
    return cells >= kLeafCells4;
}

// What to expect of a grid, in units of the constants above: the cells of four
// last-level nodes for each of D^2 where the level above has D cells along an axis
// (shapes have 0.1 to 30, most 1 to 4). Launches whose trees have less than 1
// together (and no root tape of kLeafLongTape words, the few long tapes) run word by
// word without a vote: a launch that is not picked costs 6 us with its votes.
constexpr uint32_t kLeafLongTape = 2000;
inline double leaf_load(const uint32_t* dims, uint32_t levels) {
    double above = 1.0;
    for (uint32_t l = 0; l + 1 < levels; l++) above *= dims[l];
    const double last = dims[levels - 1];
    return 4.0 * above * above * last * last * last / (double)(last == 4.0 ? kLeafCells4 : kLeafCells8);
}

}  // namespace frep
