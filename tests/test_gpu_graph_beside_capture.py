"""Stepping a small plain FP64 grid, whose steps are captured into a graph of the solver's own, while the
caller captures something else on another stream: both work, in the same thread and in another one."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["thread_local", "relaxed", "global"])
@pytest.mark.parametrize("other_thread", [False, True])
def test_steps_beside_a_capture(hteno_lib, cuda, mode, other_thread):
    from hteno import ic

    h, torch = hteno_lib, cuda
    q = ic.four_quadrant(48, 40, 5)
    with h.Solver(h.config(dims=2, nx=48, ny=40)) as a, h.Solver(h.config(dims=2, nx=48, ny=40)) as b:
        a.set_state(q)
        a.step(10)
        b.set_state(q)
        st, x = torch.cuda.Stream(), torch.zeros(64, device="cuda")
        torch.cuda.synchronize()
        g, failed = torch.cuda.CUDAGraph(), []

        def steps():
            try:
                b.step_async(10)  # two replays of the solver's graph and two plain steps
            except h.HtenoError as e:
                failed.append(e)

        with torch.cuda.graph(g, stream=st, capture_error_mode=mode):
            x.add_(1)
            if other_thread:
                t = threading.Thread(target=steps)
                t.start()
                t.join()
            else:
                steps()
            x.add_(1)
        g.replay()
        b.sync()
        torch.cuda.synchronize()
        assert not failed
        assert (x == 2).all() and a.time() == b.time()
        np.testing.assert_array_equal(a.get_state(), b.get_state())
