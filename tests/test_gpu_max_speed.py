"""The first dt of a new state: the largest wave speed, in double, where cells below the largest speed
found so far are only bounded in float.  Against numpy's doubles, over magnitudes, signs and NaN."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def state(kind, nx, ny, seed=3):
    rng = np.random.default_rng(seed)
    q = np.empty((4, ny, nx))
    q[0] = rng.uniform(0.1, 2.0, (ny, nx))
    q[1:3] = rng.normal(size=(2, ny, nx))
    q[3] = rng.uniform(2.0, 9.0, (ny, nx)) + (q[1] ** 2 + q[2] ** 2) / q[0]
    if kind == "wide":  # magnitudes beyond what a float holds, negative densities and pressures
        q *= 10.0 ** rng.integers(-60, 60, (1, ny, nx)) * rng.choice([-1.0, 1.0], q.shape)
    elif kind == "cold":  # nearly no pressure: e - ke cancels
        q[3] = (0.5 * (q[1] ** 2 + q[2] ** 2) / q[0]) * (1.0 + 1e-9 * rng.normal(size=(ny, nx)))
    elif kind == "flat":  # every cell within a few ulps of every other
        q[:] = np.array([1.0, 0.3, -0.2, 2.5])[:, None, None] * (1 + 1e-15 * rng.integers(-3, 4, q.shape))
    elif kind == "odd":  # NaN in one component, vanishing and huge densities, a lone fast cell
        q[rng.integers(0, 4, 5), rng.integers(0, ny, 5), rng.integers(0, nx, 5)] = np.nan
        q[0, 0, 0], q[0, 1, 1] = 1e-300, 1e300
        q[1, ny - 1, nx - 1] = 7e4
    return q


def first_dt(q, dx, dy, cfl=0.5, gamma=1.4):
    with np.errstate(all="ignore"):
        u, v = q[1] / q[0], q[2] / q[0]
        p = (q[3] - 0.5 * (q[1] * u + q[2] * v)) * (gamma - 1.0)
        c = np.sqrt(np.abs(gamma * p / q[0]))
        m = np.fmax(np.fmax(u - c, np.abs(u + c)), np.fmax(v - c, np.abs(v + c)))
    return cfl * min(dx, dy) / np.nanmax(m)


# one block, ragged, more cells than one pass of the grid
@pytest.mark.parametrize("nx,ny", [(6, 9), (61, 47), (1301, 1003)])
@pytest.mark.parametrize("kind", ["plain", "wide", "cold", "flat", "odd"])
def test_first_dt(hteno_lib, cuda, nx, ny, kind):
    h = hteno_lib
    q = state(kind, nx, ny)
    cfg = dict(dims=2, nx=nx, ny=ny, precision=h.PREC_MIXED)
    c = h.config(**cfg)
    want = first_dt(q, (c.xr - c.xl) / nx, (c.yt - c.yb) / ny, c.cfl, c.gamma)
    with h.Solver(h.config(**cfg)) as s:
        s.set_state(q)
        s.step(1)
        assert s.time()[0] == want
    with h.Batch([h.config(**cfg), h.config(**cfg)]) as b:
        b.set_state(0, q[:, ::-1].copy())
        b.set_state(1, q)
        b.step(1)
        assert b.time(0)[0] == want and b.time(1)[0] == want
    # the Hermite kernel may contract its products: the pressure's rounding, amplified where it cancels
    with h.Solver(h.config(scheme=h.SCHEME_HERMITE, **cfg)) as s:
        s.set_state(q)
        s.step(1)
        tol = 1e-6 if kind == "cold" else 1e-14
        assert abs(s.time()[0] - want) <= tol * want
