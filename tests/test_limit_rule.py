"""Launch shape of the Hermite 2D limiter (limit_rule.h): a line's segments follow from its own length,
whatever the other side of the grid, and a block is whole warps."""
from __future__ import annotations

import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "hermite-teno_gb300" / "csrc"


def test_segments_follow_the_line(tmp_path):
    src = tmp_path / "rule.cpp"
    src.write_text('#include <cstdio>\n#include "limit_rule.h"\nint main() {\n'
                   "  const int sides[] = {6, 31, 40, 47, 48, 111, 112, 300, 1000, 2048};\n"
                   "  for (int nx : sides)\n    for (int ny : sides) {\n"
                   "      const hteno::LimitShape s = hteno::limit_shape(nx, ny);\n"
                   '      std::printf("%d %d %d %d %d\\n", nx, ny, s.lines, s.segx, s.segy);\n    }\n}\n')
    exe = tmp_path / "rule"
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    rows = [[int(x) for x in ln.split()] for ln in
            subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()]
    of = {}
    for nx, ny, lines, segx, segy in rows:
        assert of.setdefault(nx, segx) == segx and of.setdefault(ny, segy) == segy
        assert lines * max(segx, segy) % 32 == 0 and lines * max(segx, segy) <= 256
        for n, segs in ((nx, segx), (ny, segy)):
            assert 2 <= segs <= 8 and (segs == 2 or n // segs >= 12) and (n < 112 or segs == 8)


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(6, 300), (300, 6), (47, 400), (1000, 48)])
def test_uneven_sides_bitwise(hteno_lib, cuda, oracle, nx, ny):
    """Different numbers of segments in the two directions, threads past the shorter one's among them."""
    from test_gpu_limiter import data2d, run2

    q, v, w = data2d(nx, ny, "noise")
    want = oracle.hermite2d_run(q, v, w, 2)[:3]
    for a, b in zip(run2(hteno_lib, q, v, w, 2), want):
        np.testing.assert_array_equal(a, b)
