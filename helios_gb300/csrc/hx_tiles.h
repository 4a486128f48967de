// Tile candidate of a contraction level that the tile table has no entry for
// (host code, kept apart from the kernels so that it can be tested alone).
#pragma once

namespace tc {

// What the choice goes by: ceil log2 of the widest N, floor log2 of the
// multiply-adds, and the mean K of the level's products weighted by their
// outputs -- the multiply-adds per output, which tell how much of a tile's
// time is its k-loop and how much its drain and epilogue.
struct LevelShape {
    int n_class, work_class;
    double k_per_output;
};

// The default candidate (0), or the mode's last one for large levels of long
// K: a pair of CTAs for LOW (3 slices) and HIGH (5), four stages of half the
// depth for MID (4). EXACT (7) has no such candidate. Against candidate 0, over
// the levels of polyenes of 96 to 192 sites and ladders of 64 and 80: with
// 2080 or more per output (and 2^36 multiply-adds, N above 2048) the pairs take
// 0.87 to 0.99 of its time, and MID's last 0.94 to 1.01; a pair takes 1.05 to 1.19
// at 1120 to 1720 per output (a level of one long product and three of K = N) and
// 1.16 to 1.43 at K = 192, where MID's last takes 0.95 to 0.97 and 1.00.
constexpr double kPairK = 2048.0, kDeepK = 1024.0;
inline int fallback_candidate(int mode, int candidates, const LevelShape &s)
{
    if (mode > 2 || s.n_class < 12 || s.work_class < 36) return 0;
    return s.k_per_output >= (mode == 1 ? kDeepK : kPairK) ? candidates - 1 : 0;
}

// A candidate of a mode (its tiles take `ctas` CTAs each) on a device that
// holds `clusters` pairs of them at once: the default one instead of a pair
// that does not fit, -1 (an error) where the caller asked for it by number.
inline int held_candidate(int candidate, int ctas, int clusters, bool forced)
{
    if (ctas == 1 || clusters > 0) return candidate;
    return forced ? -1 : 0;
}

}  // namespace tc
