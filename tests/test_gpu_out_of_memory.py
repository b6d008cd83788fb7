"""Calls that find no device memory fail with an error, and work once there is
some: an array whose allocation failed is empty, not there without memory."""
import numpy as np
import pytest

import parity_cases as PC

pytestmark = pytest.mark.gpu


class Hold:
    """All device memory but `leave` bytes, while it lasts."""

    def __init__(self, leave):
        self.leave = leave

    def __enter__(self):
        import torch
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        self.block = torch.empty(torch.cuda.mem_get_info()[0] - self.leave, dtype=torch.uint8, device="cuda")

    def __exit__(self, *_):
        import torch
        del self.block
        torch.cuda.empty_cache()


def test_adjoint_tape(fundem):
    sc = PC.pour_mm(n=64)
    rng = np.random.default_rng(3)
    w, u = rng.standard_normal((2, 64, 3))

    def run(tight):
        s = fundem.Simulation.from_scenario(sc, records=False)
        s.detect()
        s.adjoint_begin(2000)       # a tape of 2,000 steps: some 400 MB
        s.adjoint_forward(20)
        s.sync()
        if tight:
            for _ in range(2):
                with Hold(100 << 20):
                    with pytest.raises(fundem.FundemError):
                        s.adjoint_backward(w, u)
        out = s.adjoint_backward(w, u)
        s.adjoint_end()
        s.step(1)
        s.sync()
        s.close()
        return out

    ref, got = run(False), run(True)
    for a, b in zip(ref, got):
        assert np.abs(a - b).max() <= 1e-12 * np.abs(a).max()   # the sweep adds with atomics
