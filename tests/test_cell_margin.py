"""The margin of a search grid's cells (sm_grid.h cell_slack): a point lies within it of the cell that
its rounded coordinate names, wherever the cloud lies and however fine the cells, and it never passes
half a cell, so that a search looks at a few rings of cells. CPU only."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <random>
#include "sm_grid.h"
int main() {
    std::mt19937 rng(3);
    auto         uni = [&]() { return std::uniform_real_distribution<double>(0.0, 1.0)(rng); };
    for (int dim : {1, 100, 20000, 300000, (1 << 20) - 1}) {
        if (!(smg::cell_slack(dim) <= 0.5f && smg::cell_slack(dim) >= smg::kCellSlack))
            std::printf("dim %d: margin %g\n", dim, smg::cell_slack(dim));
        for (double off : {0.0, 1e5, 3e6, 2e8, 1e12})
            for (int t = 0; t < 20000; t++) {
                const float g = (float)(0.1 + uni()), org = (float)((uni() < 0.5 ? -off : off) + uni());
                const float x = (float)((double)org + uni() * dim * (double)g);
                if (x < org || !(((double)x - org) / g < dim))
                    continue;
                const int    c = smg::coord(x, org, g, dim);
                const double u = ((double)x - org) / g, m = smg::cell_slack(dim);
                if (u < c - m || u > c + 1 + m)
                    std::printf("dim %d off %g: %.9g in cell %d\n", dim, off, u, c);
            }
    }
    std::printf("done\n");
}
"""


def test_points_lie_within_the_margin_of_their_cells(tmp_path):
    src, exe = tmp_path / "margin.cpp", tmp_path / "margin"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "surface_match_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout
    assert out == "done\n", out
