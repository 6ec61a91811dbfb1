"""Small tiles of the mixed FV 2D stage and its early launches: the bits of the largest tile, for grids
smaller than a tile, ragged ones and ones with interior (TMA staged) tiles; a captured run of steps."""
from __future__ import annotations

import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(h, q, tile, steps, **kw):
    os.environ["HTENO_FV2D_TILE"] = str(tile)
    try:
        with h.Solver(h.config(dims=2, nx=q.shape[2], ny=q.shape[1], precision=h.PREC_MIXED, **kw)) as s:
            s.set_state(q)
            s.step(steps)
            return s.get_state(), s.time()[:2], s.counters()["tma_tiles"]
    finally:
        os.environ.pop("HTENO_FV2D_TILE", None)


@pytest.mark.parametrize("nx,ny", [(6, 6), (7, 9), (8, 8), (17, 33), (96, 80)])
@pytest.mark.parametrize("bc,flux,recon", [(0, 1, 0), (1, 0, 1), (0, 0, 4)])
def test_small_tiles_same_bits(hteno_lib, cuda, nx, ny, bc, flux, recon):
    from hteno import ic

    q = ic.four_quadrant(nx, ny, 11)
    want, t, _ = run(hteno_lib, q, 0, 6, bc=bc, flux=flux, recon=recon)
    for tile in (8, 9, 10, 11):
        got, tg, tma = run(hteno_lib, q, tile, 6, bc=bc, flux=flux, recon=recon)
        np.testing.assert_array_equal(got, want)
        assert tg == t and (tma > 0) == ((nx, ny) == (96, 80))  # (an interior tile, nx even)


def test_captured_steps(hteno_lib, cuda):
    """Steps recorded into a graph (plain launches there) and replayed: the bits of the same steps."""
    from hteno import ic

    h = hteno_lib
    q = ic.four_quadrant(96, 80, 5)
    cfg = dict(dims=2, nx=96, ny=80, precision=h.PREC_MIXED)
    with h.Solver(h.config(**cfg)) as a, h.Solver(h.config(**cfg)) as b:
        a.set_state(q)
        a.step(6)
        st = cuda.cuda.Stream()
        b.set_stream(st.cuda_stream)
        b.set_state(q)
        b.step(2)
        g = cuda.cuda.CUDAGraph()
        with cuda.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
            b.step_async(2)
        for _ in range(2):
            g.replay()
        cuda.cuda.synchronize()
        assert a.time()[:2] == b.time()[:2]
        np.testing.assert_array_equal(a.get_state(), b.get_state())
