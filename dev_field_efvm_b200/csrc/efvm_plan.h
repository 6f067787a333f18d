// efvm_plan.h — the rules that lay out a stage kernel's launch: rows per warp and
// whether a case runs the face-parallel kernel.  Plain host arithmetic, without
// CUDA, so that it can be compiled and checked on its own.
#pragma once

#include <algorithm>

namespace efvm {

constexpr int GRID_Y_MAX = 65535;  // blocks along a launch's y
// Rows of a tile of the face-parallel kernel (efvm_tile.cu).
constexpr int TILE_ROWS = 3;

// Rows each warp marches: the count in [lo, hi] whose blocks, dealt to the resident
// slots in order, finish first.  A block of r rows takes r passes, one more that
// only forms the face below its first row (about half a pass), and the column's
// last block is shorter.  A count that leaves a few full blocks for one more wave
// pays for nearly two: by the fewest-rows rule that this one replaces 1024^2 took
// 12 rows and 1.05 waves (us per step 193 -> 159), 4400x820 viscous 804 -> 742.
// In 3-D short last blocks fill the gaps the long ones leave (tail_cost 0.15:
// over nine cases of 50 to 256 cells a side the choice is within 0.9 % of the best
// of 2..16 rows on average, 3 % at most; without it 1.7 and 6 %); in 2-D the same
// term made 1024^2 5 % and 4096^2 3 % slower.
//
// The blocks of a column lie along the launch's y, so a tall grid takes at least
// the rows that fit its column there (ny = 900,000 at six blocks per SM: by cost
// alone 13 rows, 69,231 blocks).
inline int pick_rows(long long across, int ny, long long slots, int lo, int hi, double tail_cost) {
    lo = std::min(hi, std::max(lo, (ny + GRID_Y_MAX - 1) / GRID_Y_MAX));
    int best = lo;
    double best_cost = 1e300;
    for (int rows = lo; rows <= hi; ++rows) {
        const int down = (ny + rows - 1) / rows, tail = ny - (down - 1) * rows;
        const long long blocks = across * down, full = blocks / slots, over = blocks - full * slots;
        const double last = over == 0 ? 0.0 : (over <= across ? tail + 0.5 : rows + 0.5);
        const double cost = (double)full * (rows + 0.5) + last + tail_cost * (tail + 0.5);
        if (cost < best_cost) {
            best_cost = cost;
            best = rows;
        }
        if (rows >= ny) break;
    }
    return best;
}

// Whether an FP64 case without explicit form, rows and blocks runs the face-parallel
// kernel: up to a number of cells, and where its column of tiles fits the launch.
// The lines lie where the forms measured equal (us per step, other form /
// face-parallel): against the TMA-fed form 512^2 57.5 / 53.9, 768^2 95.7 / 106,
// 1003x777 121 / 140; against the viscous strip form 1500x279 113 / 105, 2200x410
// 203 / 203.
constexpr long long TILE_CELLS_TMA = 400000, TILE_CELLS_STRIP = 800000;
inline bool tile_fits(long long cells, int ny, bool tma_applies) {
    return cells <= (tma_applies ? TILE_CELLS_TMA : TILE_CELLS_STRIP) && (ny + TILE_ROWS - 1) / TILE_ROWS <= GRID_Y_MAX;
}

}  // namespace efvm
