// efvm_plan.h — the rules that lay out a stage kernel's launch: rows per warp and
// whether a case runs the face-parallel kernel.  Plain host arithmetic, without
// CUDA, so that it can be compiled and checked on its own.
#pragma once

#include <algorithm>

namespace efvm {

constexpr int GRID_Y_MAX = 65535;  // blocks along a launch's y
// Rows of a tile of the face-parallel kernel (efvm_tile.cu).
constexpr int TILE_ROWS = 3;

// When the last block of a stage ends, in half passes, if `slots` blocks run at a time
// and each free slot takes the next one.  A block of r rows takes r passes and one
// more that only forms the face below its first row (about half a pass); `across`
// blocks lie side by side, and the last ones of the columns, launched last, are
// shorter and fill the slots that the full ones leave free.
inline long long stage_end(long long across, int ny, long long slots, int rows) {
    const int down = (ny + rows - 1) / rows;
    const long long full = 2LL * rows + 1, tail = 2LL * (ny - (down - 1) * rows) + 1;
    const long long blocks = across * (down - 1), begun = blocks / slots * full, over = blocks % slots;
    auto ceil_div = [](long long x, long long y) { return x > 0 ? (x + y - 1) / y : 0; };
    if (over == 0) return begun + ceil_div(across, slots) * tail;
    // `over` slots run one more full block; the others take tails from `begun` on
    const long long idle = slots - over;
    if (ceil_div(across, idle) * tail <= full) return begun + full;
    const long long before = full / tail, past = ceil_div(full, tail);
    const long long on_idle = std::max(past, ceil_div(across + over * past, slots)) * tail;
    const long long on_last = full + ceil_div(across - idle * before, slots) * tail;
    return begun + std::min(on_idle, on_last);
}

// Rows each warp marches, in [lo, hi]: the fewest whose blocks fit the resident slots
// at once, unless another count ends the stage at least 8 % earlier by stage_end.
// The fewest-rows rule alone pays for a whole wave where it is cut off at hi or leaves
// a few blocks over: 1024^2 took 12 rows and 1.05 waves (us per step 193 -> 159),
// 4400x820 viscous 804 -> 742.  Over 120 2-D grids of 60,000 to 17 million cells,
// most of them random, in four forms the choice is 0.6 % from the best of 2..16 rows on average
// (fewest rows 7.3 %), over 68 3-D grids 0.7 % (6.0 %).  The 8 % keep the fewest rows
// where the estimate does not separate the counts: by stage_end alone 8 of 204 3-D
// cases ran 3 to 13 % slower than with the fewest rows, so 4, by up to 5 %.
//
// The blocks of a column lie along the launch's y, so a tall grid takes at least
// the rows that fit its column there.
inline int pick_rows(long long across, int ny, long long slots, int lo, int hi) {
    lo = std::min(hi, std::max(lo, (ny + GRID_Y_MAX - 1) / GRID_Y_MAX));
    const int top = std::max(lo, std::min(hi, ny));  // more rows than the grid has change nothing
    const int fewest = (int)std::min<long long>(top, std::max<long long>(lo, (across * ny + slots - 1) / slots));
    int best = fewest;
    for (int rows = lo; rows <= top; ++rows)
        if (stage_end(across, ny, slots, rows) < stage_end(across, ny, slots, best)) best = rows;
    const long long end = stage_end(across, ny, slots, best);
    return 100 * end < 92 * stage_end(across, ny, slots, fewest) ? best : fewest;
}

// Whether an FP64 case without explicit form, rows and blocks runs the face-parallel
// kernel, by its grid.  Up to one wave of tiles it always does: there a stage is one
// tile's latency (10,000 x 1 cells: 14.4 us per step against 20.5).  Above, up to a
// number of cells, which lies where the forms measured equal: 300,000 against the
// TMA-fed form (us per step, TMA-fed / face-parallel, 512^2 58 / 54, 600^2 66 / 72,
// 800 x 500 67 / 76), 815,000 against the viscous strip form (2000 x 400 171 / 162,
// 2200 x 410 203 / 203).  A tile costs the same however many of its rows the grid
// fills, and a flat grid leaves the strips' marches short as well, so the line falls
// with the cube of rows in whole tiles to rows: at ny = 1 the tiles lose from one
// wave on (60,000 cells 39 us against 28, 400,000 220 against 113), at ny = 4 from
// about 100,000 cells (400,000: 101 against 73).  Over 306 grids of 5,000 to 800,000
// cells and 1 to 9750 rows the choice is 0.4 % from the faster form on average.
constexpr int TILE_COLS = 31, TILE_BLOCKS = 4;  // a tile's columns; resident blocks per SM
constexpr long long TILE_CELLS_TMA = 300000, TILE_CELLS_STRIP = 815000;
inline bool tile_fits(int nx, int ny, bool tma_applies) {
    const int down = (ny + TILE_ROWS - 1) / TILE_ROWS;
    if (down > GRID_Y_MAX) return false;  // the column of tiles lies along the launch's y
    if ((long long)((nx + TILE_COLS - 1) / TILE_COLS) * down <= 148LL * TILE_BLOCKS) return true;
    const double f = (double)down * TILE_ROWS / ny;
    return (double)nx * ny * f * f * f <= (double)(tma_applies ? TILE_CELLS_TMA : TILE_CELLS_STRIP);
}

}  // namespace efvm
