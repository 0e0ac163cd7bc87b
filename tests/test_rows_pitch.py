"""The rule that chooses a single solve's row pitch (fdtd_gb300/csrc/rows.h),
compiled into a small host program, on the CPU."""
from __future__ import annotations

import os
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include "rows.h"
using fdtd::solve_rows_pitch;

int main()
{
    const size_t much = size_t(1) << 38, rows = 300 * 300;
    const size_t d = 73, compact = 61;  // bytes per cell
    // rows below 16 cells and multiples of 16 stay
    for (int nx : {3, 15, 16, 48, 512})
        for (int form = 0; form < 3; form++)
            if (solve_rows_pitch(nx, rows, form == 2, form == 1, form == 1 ? compact : d, much) != nx) return 1;
    // compact forms: always up to the next multiple; two-pass: never
    for (int nx : {17, 33, 61, 217})
        if (solve_rows_pitch(nx, rows, false, true, compact, much) != (nx + 15) / 16 * 16 ||
            solve_rows_pitch(nx, rows, true, false, d, much) != nx) return 2;
    // D form: up to 4/3
    for (int nx : {24, 36, 49, 217})
        if (solve_rows_pitch(nx, rows, false, false, d, much) != (nx + 15) / 16 * 16) return 3;
    for (int nx : {17, 23, 33, 35})
        if (solve_rows_pitch(nx, rows, false, false, d, much) != nx) return 4;
    // memory: a quarter of what dense rows leave free, and no wrap-around where they do not fit
    const size_t dense = rows * 17 * compact, extra = rows * 15 * compact + rows * 17 * 4;
    if (solve_rows_pitch(17, rows, false, true, compact, dense + 4 * extra) != 32) return 5;
    if (solve_rows_pitch(17, rows, false, true, compact, dense + 4 * extra - 4) != 17) return 6;
    if (solve_rows_pitch(17, rows, false, true, compact, dense - 1) != 17) return 7;
    if (solve_rows_pitch(17, rows, false, true, compact, 0) != 17) return 8;
    return 0;
}
"""


def test_pitch_rule(tmp_path):
    cuda = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))
    if shutil.which("g++") is None or not (cuda / "include" / "cuda_runtime.h").exists():
        pytest.skip("no compiler or CUDA headers")
    src, exe = tmp_path / "pitch.cpp", tmp_path / "pitch"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{ROOT / 'fdtd_gb300' / 'csrc'}", f"-I{cuda / 'include'}", str(src), "-o",
                    str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
