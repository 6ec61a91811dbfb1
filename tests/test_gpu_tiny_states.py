"""Plain FP64 at the ends of the double range, bit for bit against the oracle: states so small that a kinetic
energy's half is subnormal and rounds, and a stage combination whose doubled sum overflows by itself."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SCALES = (1e-305, 1e-307, 1e-312)


@pytest.mark.parametrize("scale", SCALES)
@pytest.mark.parametrize("nx,ny", [(40, 33), (150, 133)])
@pytest.mark.parametrize("flux", [0, 1])
def test_fv2d(hteno_lib, cuda, oracle, scale, nx, ny, flux):
    from hteno import ic

    q = np.ascontiguousarray(ic.four_quadrant(nx, ny, 3) * scale)
    want, t, n = oracle.fv2d_run(q, 4, flux=flux)
    with hteno_lib.Solver(hteno_lib.config(dims=2, nx=nx, ny=ny, flux=flux)) as s:
        s.set_state(q)
        s.step(4)
        assert s.time()[:2] == (t, n)
        np.testing.assert_array_equal(s.get_state(), want)


@pytest.mark.parametrize("scale", SCALES)
@pytest.mark.parametrize("flux", [0, 1])
def test_fv1d(hteno_lib, cuda, oracle, scale, flux):
    x = np.arange(120)
    q = np.stack([1 + 0.3 * np.sin(0.1 * x) + (x > 60), 0.4 * np.cos(0.2 * x), 4 + 0.5 * np.sin(0.05 * x)]) * scale
    q = np.ascontiguousarray(q)
    want, t, n = oracle.fv1d_run(q, 20, flux=flux)
    with hteno_lib.Solver(hteno_lib.config(dims=1, nx=120, cfl=0.5, flux=flux, recon=1)) as s:
        s.set_state(q)
        s.step(20)
        assert s.time()[:2] == (t, n)
        np.testing.assert_array_equal(s.get_state(), want)


@pytest.mark.parametrize("scale", SCALES)
def test_hermite2d(hteno_lib, cuda, oracle, scale):
    from test_gpu_limiter import data2d, run2

    q, v, w = (np.ascontiguousarray(a * scale) for a in data2d(40, 33, "noise"))
    want = oracle.hermite2d_run(q, v, w, 2)[:3]
    for a, b in zip(run2(hteno_lib, q, v, w, 2), want):
        np.testing.assert_array_equal(a, b)


def test_third_stage_overflow(hteno_lib, cuda):
    """q0 + 2 (qn + dt rhs) with a sum above 2^1023: the doubled sum is infinite, whatever q0 is."""
    qn = np.array([9.5e307, 1.7e308, -1.2e308, 8.9e307, 8.98e307, -8.99e307])
    q0 = np.array([-1.7e308, -1.7e308, 1.7e308, -1e308, 1.0, 1e308])
    a, b, z = (cuda.from_numpy(x).cuda() for x in (q0, qn, np.zeros_like(qn)))
    out = cuda.empty_like(a)
    assert hteno_lib.lib().hteno_ssprk3_batch(a.data_ptr(), b.data_ptr(), z.data_ptr(), 0.01, 3, out.data_ptr(), qn.size,
                                              None) == 0
    cuda.cuda.synchronize()
    with np.errstate(over="ignore"):
        np.testing.assert_array_equal(out.cpu().numpy(), (q0 + 2.0 * qn) / 3.0)
