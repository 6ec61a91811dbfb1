"""The Hermite limiter's segmented sweeps (Hermite 2D and 1D): the bits of the reference's one
Gauss-Seidel sweep per line whatever the length of a line, the number of segments and the data --
smooth, noisy, and tails running out into constant regions (the slowest to agree)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def data2d(nx, ny, kind, seed=5):
    from hteno import ic

    rng = np.random.default_rng(seed)
    q = ic.four_quadrant(nx, ny, seed)
    if kind == "flat":  # constant quadrants, momentum zero in two of them, lone nonzero moments
        q[1, : ny // 2] = 0.0
        q[2] = 0.0
        q[3] += 1.0
        v, w = np.zeros_like(q), np.zeros_like(q)
        for a in (v, w):
            a[:, rng.integers(0, ny, 5), rng.integers(0, nx, 5)] = rng.normal(size=(4, 5))
        v[:, :, 0] = 0.7
        w[:, 0, :] = -0.3
    else:
        v, w = rng.normal(size=q.shape) * 0.3, rng.normal(size=q.shape) * 0.3
    return tuple(np.ascontiguousarray(a) for a in (q, v, w))


def run2(h, q, v, w, nsteps, **kw):
    cfg = h.config(dims=2, scheme=h.SCHEME_HERMITE, nx=q.shape[2], ny=q.shape[1], **kw)
    with h.Solver(cfg) as s:
        s.set_state(q)
        s.set_moments(v, w)
        s.step(nsteps)
        return s.get_state(), *s.get_moments()


# a few cells; one segment row short of the next count; ragged; 32 lines a block (both launch shapes)
@pytest.mark.parametrize("nx,ny,steps", [(6, 6, 3), (31, 65, 3), (130, 97, 2), (257, 64, 2), (640, 612, 1)])
@pytest.mark.parametrize("kind", ["noise", "flat"])
def test_limiter_segments_bitwise(hteno_lib, cuda, oracle, nx, ny, steps, kind):
    q, v, w = data2d(nx, ny, kind)
    want = oracle.hermite2d_run(q, v, w, steps)[:3]
    got = run2(hteno_lib, q, v, w, steps)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("nx,ny", [(6, 6), (130, 97), (640, 612), (701, 641)])
def test_limiter_segments_mixed(hteno_lib, cuda, nx, ny):
    """Mixed precision against plain FP64 after one step on smooth data: a moment's float rounding is
    about 2^-24 |q| nx relative to |q|, a few 1e-5; cut-off flips and the stages multiply it."""
    from hteno import ic

    q = np.ascontiguousarray(ic.smooth_waves_2d(nx, ny))
    v = np.gradient(q, 1.0 / nx, axis=2)
    w = np.gradient(q, 1.0 / ny, axis=1)
    v, w = np.ascontiguousarray(v), np.ascontiguousarray(w)
    want = run2(hteno_lib, q, v, w, 1)
    got = run2(hteno_lib, q, v, w, 1, precision=hteno_lib.PREC_MIXED)
    for a, b, tol in zip(got, want, (1e-5, 1e-2, 1e-2)):
        assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)


# fewer cells than segments, one cell a segment and one more, ragged
@pytest.mark.parametrize("nx", [6, 41, 42, 85, 333, 1500])
@pytest.mark.parametrize("kind", ["noise", "flat", "waves"])
def test_hermite1d_sensor_bitwise(hteno_lib, cuda, oracle, nx, kind):
    """LMPE hits (runs of candidates of every length) and the segmented sweep, several steps, so that
    flags persist and meet new candidates."""
    rng = np.random.default_rng(nx)
    x = (np.arange(nx) + 0.5) / nx
    if kind == "waves":
        rho = 1.5 + 0.4 * np.sin(2 * np.pi * x) + np.where((x > 0.3) & (x < 0.6), 0.5, 0.0)
    elif kind == "flat":
        rho = np.where(x < 0.4, 1.0, 2.0)
    else:
        rho = rng.uniform(0.5, 2.0, nx)
    q = np.ascontiguousarray(np.stack([rho, 0.3 * rho * (kind != "flat"), 2.5 + 0.1 * rho]))
    v = rng.normal(size=q.shape) * 0.1
    if kind == "flat":
        v *= 0.0
        v[:, nx // 2] = 1.0
    v = np.ascontiguousarray(v)
    want_q, want_v, _, n = oracle.hermite1d_run(q, v, 5)
    cfg = hteno_lib.config(dims=1, scheme=hteno_lib.SCHEME_HERMITE, nx=nx)
    with hteno_lib.Solver(cfg) as s:
        s.set_state(q)
        s.set_moments(v)
        s.step(5)
        np.testing.assert_array_equal(s.get_state(), want_q)
        np.testing.assert_array_equal(s.get_moments(), want_v)
