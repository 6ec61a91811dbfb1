"""One optimiser step of the classifier: the gradient that grad() reports, Adam on the float32 master
parameters, and the BF16 images the other kernels read, from a tile short of full to two per block."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_mlp import bf16_bits, mref, random_params, to_dev  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 129, 128 * 40 + 3, 128 * 304 + 5])
def test_one_adam_step(hteno_lib, cuda, mref, n):  # noqa: F811
    rng = np.random.default_rng(n)
    _, xb = bf16_bits(rng.standard_normal((n, 6)) * 0.5, mref)
    y = rng.integers(0, 8, size=n).astype(np.uint8)
    p0 = random_params(rng, mref).astype(np.float32)
    xd, yd = to_dev(cuda, xb), to_dev(cuda, y)
    lr = 1e-2
    with hteno_lib.Mlp() as m, hteno_lib.Mlp() as k:
        m.set_params(p0)
        g, loss0 = m.grad(xd, yd)
        loss = m.train(xd, yd, epochs=1, batch=n, lr=lr)
        p1 = m.params()
        assert loss == loss0  # the same kernel, partials added in the same order
        g = g.astype(np.float64)
        mh, vh = (0.1 * g) / 0.1, (0.001 * g * g) / 0.001
        want = p0 - lr * mh / (np.sqrt(vh) + 1e-8)
        # float32: a few roundings of the step (1 - b1, the powers and 1 - power: 2^-14 in vh's) and one
        # of the parameter
        np.testing.assert_allclose(p1, want, rtol=2.0**-23, atol=lr * 2.0**-13)
        # the images are those of the new parameters
        out = [cuda.empty((n, 3), dtype=cuda.float32, device="cuda") for _ in range(2)]
        m.predict(xd, out[0])
        k.set_params(p1)
        k.predict(xd, out[1])
        assert cuda.equal(out[0], out[1])
        assert np.array_equal(m.grad(xd, yd)[0], k.grad(xd, yd)[0])
