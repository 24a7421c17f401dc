"""The search of a spline cell (agama_b200/csrc/grid_cells.h) built for the host: the segment of
math::binSearch (src/math_core.cpp:251-280) with a bounded number of loads, on grids of any spacing
(CPU, no GPU)."""
import os
import subprocess

from conftest import ROOT


def test_cell_search(tmp_path):
    exe = str(tmp_path / "cell_search_check")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-Wno-unknown-pragmas", "-x", "c++",
                        "-I" + os.path.join(ROOT, "agama_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "cell_search_check.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and "mismatches 0" in out.stdout, out.stdout + out.stderr
