"""The one-launch stages of plain FP64 FV 1D: block edges, both block sizes, both boundaries and
fluxes, runs of graph-replayed and single steps, and the stop at t_final, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# fewest cells; around a block's 3 cells; the last size of 4-face blocks and the first of 16-face ones
@pytest.mark.parametrize("nx", [6, 7, 8, 100, 1824, 1825, 2003])
@pytest.mark.parametrize("bc,flux,recon", [(0, 1, 0), (1, 0, 1), (0, 1, 2), (1, 1, 4)])
def test_fv1d_stages_bitwise(hteno_lib, cuda, oracle, nx, bc, flux, recon):
    rng = np.random.default_rng(nx)
    x = (np.arange(nx) + 0.5) / nx
    rho = np.where(x < 0.5, 1.0, 0.3) + 0.05 * rng.uniform(size=nx) * (np.abs(x - 0.5) < 0.2)
    u = 0.2 * np.sin(2 * np.pi * x)
    q = np.ascontiguousarray(np.stack([rho, rho * u, 2.5 * np.where(x < 0.5, 1.0, 0.2) + 0.5 * rho * u * u]))
    want, t, n = oracle.fv1d_run(q, 19, bc=bc, flux=flux, recon=recon)
    cfg = hteno_lib.config(dims=1, nx=nx, cfl=0.5, bc=bc, flux=flux, recon=recon)
    with hteno_lib.Solver(cfg) as s:
        s.set_state(q)
        s.step(19)  # 16 steps as one graph, 3 single ones
        assert s.time()[:2] == (t, n)
        np.testing.assert_array_equal(s.get_state(), want)


def test_fv1d_stages_stop_and_go_on(hteno_lib, cuda, oracle):
    """A step clipped to t_final, idle steps past it, then on to a later stop."""
    from hteno import ic

    q = ic.sod(100)
    t1, t2 = 0.031, 0.05
    a, ta, na = oracle.fv1d_run(q, 10000, t_final=t1, flux=1, recon=0)
    with hteno_lib.Solver(hteno_lib.config(dims=1, nx=100, cfl=0.5, flux=1, recon=0)) as s:
        s.set_state(q)
        s.step_async(200, t1)
        s.sync()
        assert s.time()[:2] == (ta, na)
        np.testing.assert_array_equal(s.get_state(), a)
        s.step(10000, t2)
        assert abs(s.time()[0] - t2) <= 1e-15
        assert s.launches_per_step() == 3
