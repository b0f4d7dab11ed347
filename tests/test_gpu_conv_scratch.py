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


@pytest.mark.parametrize("c,k,hw", [(24, 18, 5), (20, 20, 3), (3, 17, 7), (40, 64, 3)])
def test_output_at_any_address(c, k, hw):
    """Images one by one into the rows of a larger output tensor: rows of k * hw * hw bytes, in a buffer at an odd address."""
    from nart_b200 import ops
    from nart_b200._lib import check, lib
    n = 4
    x = torch.randint(0, 256, (n, hw, hw, c), device="cuda", dtype=torch.uint8)
    plan = _plan(c, k, hw)
    want = _plan(c, k, hw, algo=ops.ALGO_DIRECT)(x)
    row = k * hw * hw
    for shift in (0, 1, 4):
        y = torch.full((n * row + shift + 1,), 7, device="cuda", dtype=torch.uint8)
        torch.cuda.synchronize()
        for i in range(n):
            check(lib.b200_conv2d_run(plan._h, x[i:i + 1].data_ptr(), 1, y.data_ptr() + shift + i * row, None))
        torch.cuda.synchronize()
        assert torch.equal(y[shift:shift + n * row].view(n, hw, hw, k), want)
        assert int(y[-1]) == 7 and (shift == 0 or int(y[0]) == 7)
