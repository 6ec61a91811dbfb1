"""Plain FP64 FV 2D with 8 lanes per face (small grids) and one thread per face (larger ones): both
sides of the rule's line, bit for bit against the oracle, over fluxes, reconstructions, boundaries."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# fewest cells, odd sides, long and thin, the last sizes below and the first above the line
@pytest.mark.parametrize("nx,ny", [(6, 6), (7, 33), (6, 400), (84, 85), (86, 85), (301, 23), (331, 21), (332, 22)])
@pytest.mark.parametrize("bc,flux,recon", [(0, 1, 0), (1, 0, 1), (0, 0, 0), (1, 1, 2), (0, 1, 4)])
def test_fv2d_lanes_bitwise(hteno_lib, cuda, oracle, nx, ny, bc, flux, recon):
    from hteno import ic

    q = ic.four_quadrant(nx, ny, 3)
    want, t, n = oracle.fv2d_run(q, 4, bc=bc, flux=flux, recon=recon)
    with hteno_lib.Solver(hteno_lib.config(dims=2, nx=nx, ny=ny, bc=bc, flux=flux, recon=recon)) as s:
        s.set_state(q)
        s.step(4)
        assert s.time()[:2] == (t, n)
        np.testing.assert_array_equal(s.get_state(), want)


@pytest.mark.parametrize("bc", [2, 3])
def test_fv2d_lanes_ghost_rows(hteno_lib, cuda, oracle, bc):
    """Boundaries whose ghosts are not copies: the transverse GL3 reads the ghost face rows."""
    from hteno import ic

    nx, ny = 40, 24
    box = dict(xl=0.0, xr=0.25, yb=0.0, yt=1.0) if bc == 2 else dict(xl=0.0, xr=4.0, yb=0.0, yt=1.0)
    q = (ic.rayleigh_taylor if bc == 2 else ic.double_mach)(nx, ny)
    want, t, n = oracle.fv2d_run(q, 6, bc=bc, flux=1, recon=0, **box)
    with hteno_lib.Solver(hteno_lib.config(dims=2, nx=nx, ny=ny, bc=bc, flux=1, recon=0, **box)) as s:
        s.set_state(q)
        s.step(6)
        np.testing.assert_array_equal(s.get_state(), want)
