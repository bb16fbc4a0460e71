"""Calls where device memory is short (needs a B200)."""
import numpy as np
import pytest

from titan_b200.host import synthetic
from titan_b200.host.system import initial_state

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps
MIB = 1 << 20


def context(deck, h0):
    from titan_b200.native import GreenGPU
    g = GreenGPU(0)
    g.setup(deck, h0)
    return g


class filled_device:
    """Leaves `free` bytes of the device's memory to the calls inside."""

    def __init__(self, free):
        self.free = free

    def __enter__(self):
        import torch
        torch.cuda.empty_cache()
        left = torch.cuda.mem_get_info(0)[0]
        assert left > self.free
        self.block = torch.empty(left - self.free, dtype=torch.uint8, device="cuda:0")

    def __exit__(self, *exc):
        import torch
        del self.block
        torch.cuda.empty_cache()


def test_a_call_after_one_that_ran_out_of_memory():
    """The failed call reports TG_ERR_NOMEM; what is called next is not touched by it."""
    from titan_b200.native import GreenGPU, TitanGPUError
    g = GreenGPU(0)
    rng = np.random.default_rng(2)
    x = rng.standard_normal((8, 8)) + 1j * rng.standard_normal((8, 8))
    want = np.linalg.solve(np.eye(8) + x @ x, x)
    g.dyson(x, x)   # (loads the kernels)
    with filled_device(64 * MIB):
        with pytest.raises(TitanGPUError) as err:
            g.dyson(np.eye(1600, dtype=complex), np.eye(1600, dtype=complex))
        assert err.value.code == -5
        assert np.allclose(g.dyson(x, x), want, rtol=0, atol=1e-12 * np.abs(want).max())
    g.close()
