"""The rules that lay out a stage kernel's launch (csrc/efvm_plan.h), compiled and
run on the host: a column of blocks fits the 65,535 blocks that a launch takes
along y for every height that the rows allow, and no grid whose column of
face-parallel tiles does not fit is sent to that kernel; the estimate behind the
rows equals dealing the blocks out one by one."""
from __future__ import annotations

import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cstdio>
#include <queue>
#include <vector>
#include "efvm_plan.h"
using namespace efvm;
// the same end by taking the blocks in order, each to the slot that is free first
static long long dealt(long long across, int ny, long long slots, int rows) {
    const int down = (ny + rows - 1) / rows;
    std::priority_queue<long long, std::vector<long long>, std::greater<long long>> free_at;
    for (long long s = 0; s < slots; ++s) free_at.push(0);
    long long end = 0;
    for (int d = 0; d < down; ++d)
        for (long long b = 0; b < across; ++b) {
            const int r = d + 1 < down ? rows : ny - (down - 1) * rows;
            const long long t = free_at.top() + 2 * r + 1;
            free_at.pop();
            free_at.push(t);
            if (t > end) end = t;
        }
    return end;
}
int main() {
    for (int across = 1; across <= 90; across += across < 12 ? 1 : 13)
        for (int ny = 1; ny <= 230; ny += ny < 40 ? 1 : 19)
            for (int slots : {1, 7, 40, 592})
                for (int rows = 1; rows <= 16; ++rows)
                    if (stage_end(across, ny, slots, rows) != dealt(across, ny, slots, rows))
                        return std::printf("end %d %d %d %d\n", across, ny, slots, rows), 1;
    // a choice never ends later than the fewest rows that fit the slots at once
    for (int across : {1, 5, 33, 577, 3000})
        for (int ny = 1; ny <= 900; ny += 7) {
            const int r = pick_rows(across, ny, 888, 2, 16);
            long long f = (across * (long long)ny + 887) / 888;
            f = f < 2 ? 2 : (f > 16 ? 16 : f);
            if (stage_end(across, ny, 888, r) > stage_end(across, ny, 888, (int)f)) return std::printf("fewest\n"), 1;
        }
    // 2-D: one block of strips across, each resident-block count, rows in [2, 16]
    for (int per_sm = 5; per_sm <= 8; ++per_sm)
        for (int ny = 1; ny <= 16 * GRID_Y_MAX; ny += ny < 800000 ? 97 : 1) {
            const int r = pick_rows(1, ny, 148LL * per_sm, 2, 16);
            if (r < 2 || r > 16 || (ny + r - 1) / r > GRID_Y_MAX) return std::printf("2-D %d %d %d\n", per_sm, ny, r), 1;
        }
    for (int across = 1; across <= 8; ++across)  // 3-D, rows in [2, 16]
        for (int ny = 1; ny <= 16 * GRID_Y_MAX; ny += ny < 600000 ? 97 : 7) {
            const int r = pick_rows(across, ny, 592, 2, 16);
            if (r < 2 || r > 16 || (ny + r - 1) / r > GRID_Y_MAX) return std::printf("3-D %d %d %d\n", across, ny, r), 1;
        }
    // past every height: still within [lo, hi] (the launch then fails with an error)
    if (pick_rows(1, 2000000, 740, 2, 16) != 16) return std::printf("past\n"), 1;
    for (int tma = 0; tma < 2; ++tma) {
        if (!tile_fits(1, 196605, tma) || tile_fits(1, 196606, tma)) return std::printf("tall\n"), 1;
        const int n = (tma ? 300000 : 815000) / 1200;  // rows in whole tiles
        if (!tile_fits(n, 1200, tma) || tile_fits(n + 1, 1200, tma)) return std::printf("cells\n"), 1;
        // one row: up to 592 tiles of 31 columns
        if (!tile_fits(592 * 31, 1, tma) || tile_fits(tma ? 592 * 31 + 1 : 40000, 1, tma)) return std::printf("flat\n"), 1;
    }
    return 0;
}
"""


def test_launch_extents_hold_for_every_height(tmp_path):
    src, exe = tmp_path / "plan.cpp", tmp_path / "plan"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "dev_field_efvm_b200", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("ny", [196605, 196606, 200000])
@pytest.mark.parametrize("viscous", [0, 1])
def test_tall_grids_step(ny, viscous):
    """nx = 2, on both sides of the line: whole steps equal the strip form's at explicit
    rows (bit for bit without viscous terms, 2e-13 of each variable's scale with)."""
    import numpy as np

    from dev_field_efvm_b200 import abi, cases
    from dev_field_efvm_b200.device import Context

    bcs = {s: abi.BC_PERIODIC for s in (abi.XLO, abi.XHI, abi.YLO, abi.YHI)}
    grid = abi.make_grid(2, ny, hi=(2.0, float(ny), 1.0), bcs=bcs | {abi.ZLO: abi.BC_SLIP_WALL, abi.ZHI: abi.BC_SLIP_WALL})
    params = abi.make_params(cfl=0.3, r_gas=1.0, reconstruction=abi.RECON_MUSCL, viscous=viscous, mu=1e-3,
                             viscosity_model=abi.VISC_CONSTANT)
    rng = np.random.default_rng(ny)
    f = rng.uniform(-1.0, 1.0, (4, ny, 2))
    u = cases.prim_to_cons(1.0 + 0.1 * f[0], 0.2 * f[1], 0.2 * f[2], 1.0 + 0.1 * f[3])
    out = []
    for form, rows in ((abi.STAGE_AUTO, 0), (abi.STAGE_STRIP, 16)):
        c = Context(grid, params)
        c.set_stage_tiling(form, rows)
        c.upload(u)
        c.step(1)
        c.step(2)
        out.append(c.download())
        c.close()
    err = np.max(np.abs(out[0] - out[1]) / np.array([1.0, 1.0, 1.0, 1.0, 3.0]))
    assert err < 2e-13 if viscous else np.array_equal(out[0], out[1])
    assert not np.array_equal(out[0], u)
