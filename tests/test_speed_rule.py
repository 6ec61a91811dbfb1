"""The largest wave speed of a new state: which grids take every cell and which filter (speed_rule.h),
and the first dt on both sides of the lines."""
from __future__ import annotations

import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "hermite-teno_gb300" / "csrc"


def test_small_grids_are_not_filtered(tmp_path):
    src = tmp_path / "rule.cpp"
    src.write_text('#include <cstdio>\n#include "speed_rule.h"\nint main() {\n'
                   "  const long cells[] = {36, 1600, 160000, 196608, 196609, 311364, 458752, 458753, 1l << 31};\n"
                   "  for (long c : cells)\n    for (int p = 0; p < 2; ++p) {\n"
                   "      const hteno::SpeedLaunch l = hteno::speed_launch(c, p);\n"
                   '      std::printf("%ld %d %d %u\\n", c, p, int(l.filter), l.blocks);\n    }\n}\n')
    exe = tmp_path / "rule"
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    for ln in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines():
        cells, prims, filtered, blocks = (int(x) for x in ln.split())
        assert filtered == (cells > (458752 if prims else 196608))
        assert blocks == min(1216, -(-cells // 256)) if filtered else blocks * 256 >= cells > blocks * 256 - 256


@pytest.mark.gpu
@pytest.mark.parametrize("scheme,n", [(0, 443), (0, 444), (1, 677), (1, 678)])
@pytest.mark.parametrize("kind", ["plain", "wide", "odd"])
def test_first_dt_about_the_lines(hteno_lib, cuda, scheme, n, kind):
    from test_gpu_max_speed import first_dt, state

    h = hteno_lib
    q = state(kind, n, n)
    cfg = h.config(dims=2, nx=n, ny=n, precision=h.PREC_MIXED, scheme=scheme)
    want = first_dt(q, 1.0 / n, 1.0 / n, cfg.cfl, cfg.gamma)
    with h.Solver(cfg) as s:
        s.set_state(q)
        if scheme:
            s.set_moments(np.zeros_like(q), np.zeros_like(q))
        s.step(1)
        # the same doubles; the Hermite kernel may contract its products
        assert abs(s.time()[0] - want) <= (1e-14 if scheme else 0.0) * want
