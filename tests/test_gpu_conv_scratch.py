"""Convolution plans that run through scratch tensors (channel counts that are no multiple of 16, 4-channel images)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _plan(c, k, hw, seed=0, **kw):
    from nart_b200 import ops
    rng = np.random.default_rng(seed)
    wt = rng.integers(0, 256, (k, c, 1, 1), dtype=np.uint8)
    bias = rng.integers(-4096, 4097, k).astype(np.int32)
    return ops.Conv2d(wt, bias, in_hw=(hw, hw), ialpha=0.02, izp=120, walpha=rng.uniform(0.002, 0.01, k).astype(np.float32),
                      oalpha=float(0.02 * 0.006 * 74 * 73 * np.sqrt(c) / 45), ozp=99, **kw)


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_plan_destroyed_while_another_device_is_current():
    """The scratch tensor goes back to the memory pool only when its own device has finished with it."""
    from nart_b200 import ops
    n, hw = 40, 56
    with torch.cuda.device(1):
        x = torch.randint(0, 256, (n, hw, hw, 24), device="cuda:1", dtype=torch.uint8)
        other = torch.randint(0, 256, (n, hw, hw, 24), device="cuda:1", dtype=torch.uint8)
        want = _plan(24, 144, hw, algo=ops.ALGO_DIRECT)(x)
        torch.cuda.synchronize()
        plan = _plan(24, 144, hw)
        plan(x)
        torch.cuda.synchronize()
        got = [plan(x) for _ in range(20)]
    with torch.cuda.device(0):
        plan.close()
    with torch.cuda.device(1):
        _plan(24, 144, hw)(other)
        torch.cuda.synchronize()
        assert all(torch.equal(g, want) for g in got)
