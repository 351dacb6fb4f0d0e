// Sizes of the large splitter's levels (build.cu), plain host arithmetic.
//
// A segment of more than SPLIT_MIN points is open: it is split in two by many blocks, a
// block per tile of it.  A level's grids have to cover the tiles of all its open
// segments, which only the device knows.  Open segments hold more than SPLIT_MIN points
// each and the points of a level are at most n, so there are at most n / (SPLIT_MIN + 1)
// of them, and each has less than one tile more than its points fill.  (The largest
// job's tiles times the number of jobs, the bound before, is the same for one job; one
// job of 3M points beside 2,000 small ones got 1.1M blocks a launch for 1,500 tiles.)
#pragma once

namespace ikdg {

constexpr int SPLIT_MIN = 4096;  // larger segments are split by many blocks
constexpr int SPLIT_TILE = 2048;
// The histogram takes larger tiles: with one point per bin on average (2,048 points) a
// tile's flush was an addition in L2 per point.  2M points, nine levels: 88 -> 66 us.
constexpr int HIST_TILE = 8192;

inline long long split_segs_cap(long long n) { return n / (SPLIT_MIN + 1) + 1; }
inline long long split_tiles_cap(long long n) { return n / SPLIT_TILE + split_segs_cap(n); }
inline long long split_htiles_cap(long long n) { return n / HIST_TILE + split_segs_cap(n); }

struct SplitGrid {
    long long segs, tiles, htiles;
};
// Level `level` (0: the jobs) of a call with n points in njobs jobs.
inline SplitGrid split_grid(long long n, long long njobs, int level) {
    const long long cap = split_segs_cap(n);
    const long long s = level < 31 && (njobs << level) < cap ? njobs << level : cap;
    return SplitGrid{s, n / SPLIT_TILE + s, n / HIST_TILE + s};
}

}  // namespace ikdg
