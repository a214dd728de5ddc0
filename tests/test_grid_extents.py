"""Cell counts of the search grids (sm_grid.h) at extents beyond what an int counts: stray points,
or huge numbers in the place of missing values, are finite and belong to the cloud. CPU only."""
import subprocess

import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "sm_grid.h"
int main() {
    const float inf = 1.0f / 0.0f;
    std::printf("%d %d %d %d\n", smg::dim_of(0.0f, 1.0f), smg::dim_of(99.5f, 1.0f),
                smg::dim_of(3e9f, 1.0f), smg::dim_of(inf, inf));
    for (float e : {1e3f, 1e7f, 3e9f, 1e20f, 3e38f, inf}) {
        const float ext[3] = {e, e, 400.0f}, one[3] = {e, 400.0f, 400.0f};
        const float g[4] = {smg::thin_cell(1.0f, ext), smg::sample_cell(1.0f, one, 1ll << 25),
                            smg::query_cell(1.0f, ext), smg::query_cell(1.0f, one)};
        bool ok = smg::cells_of(ext, 1.0f) >= 1 && smg::cells_of(one, g[1]) <= (1ll << 25) &&
                  smg::cells_of(ext, g[2]) <= smg::kMaxCells &&
                  smg::cells_of(one, g[3]) <= smg::kMaxCells;
        for (float s : g)
            for (float x : {e, 400.0f})
                ok = ok && smg::dim_of(x, s) >= 1;
        ok = ok && smg::dim_of(e, g[0]) <= (1 << 20);
        // the grids' own loop (build_hgrid)
        float h = 1.0f;
        int   it = 0;
        for (; it < 1000 && smg::dim_of(e, h) >= (1 << 20); it++)
            h *= 2.0f;
        ok = ok && it < 1000 && smg::dim_of(e, h) >= 1 && smg::dim_of(e, h) * (double)h >= (e < inf ? e : 0);
        std::printf("%d\n", ok);
    }
}
"""


def test_counts_of_any_extent(tmp_path):
    src, exe = tmp_path / "extents.cpp", tmp_path / "extents"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "surface_match_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout
    lines = out.split("\n")
    assert lines[0] == f"1 100 {1 << 30} 1"
    assert lines[1:7] == ["1"] * 6, out
