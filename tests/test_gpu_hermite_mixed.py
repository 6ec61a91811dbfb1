"""Hermite 2D mixed precision: both sides of a face and pairs of cells at once in the face and flux
kernels, at sizes around a block, against the double oracle.  Tolerance: the L1 error of float faces and
fluxes that the mixed path's test at 48 x 48 allows, for density and both its moments times the cell."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(6, 6), (7, 33), (129, 6), (64, 65), (127, 128)])
def test_hermite_mixed_sizes(hteno_lib, cuda, oracle, nx, ny):
    from hteno import ic

    h = hteno_lib
    q = ic.gaussian_blobs_shock(nx, ny, 2)
    dx, dy = 1.0 / nx, 1.0 / ny
    v = np.gradient(q, dx, axis=2) * 0.5
    w = np.gradient(q, dy, axis=1) * 0.5
    want = oracle.hermite2d_run(q, v, w, 3)[:3]
    with h.Solver(h.config(dims=2, scheme=h.SCHEME_HERMITE, nx=nx, ny=ny, precision=h.PREC_MIXED)) as s:
        s.set_state(q)
        s.set_moments(v, w)
        s.step(3)
        got = (s.get_state(), *s.get_moments())
        assert s.status() == 0
    for a, b, scale in zip(got, want, (1.0, dx, dy)):
        assert np.abs(a[0] - b[0]).mean() * scale <= 1e-4
