"""b200_case_run_host on the caller's own host buffers: small pinned ones are read and written in place by the layout
kernels, whatever part of an array they are."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _logits_case(k, f32_in):
    """c inputs of one pixel -> k float logits: the shapes whose conversions move 16 bytes at a time."""
    from nart_b200.case import Case
    rng = np.random.default_rng(k)
    c = 24
    cs = Case()
    t = cs.input_f32(c, 1, 1, 0.02, 120) if f32_in else cs.input_u8(c, 1, 1)
    t = cs.ip(t, rng.integers(0, 256, (k, c), dtype=np.uint8), None, ialpha=0.02, izp=120, walpha=0.005, oalpha=0.03, ozp=111)
    cs.output_f32(t, 0.03, 111)
    cs.prepare(2)
    return cs, c


@pytest.mark.parametrize("f32_in", [True, False])
@pytest.mark.parametrize("k", [1, 10, 18, 1001])
def test_rows_of_pinned_arrays(k, f32_in):
    """Images one by one into the rows of a pinned logits array: rows of 4 k bytes, at any multiple of four."""
    cs, c = _logits_case(k, f32_in)
    rng = np.random.default_rng(3)
    n = 5
    x = rng.normal(0, 1, (n, c, 1, 1)).astype(np.float32) if f32_in else rng.integers(0, 256, (n, c, 1, 1), dtype=np.uint8)
    want = [cs.run_host([x[i:i + 1]], [(np.float32, (k,))])[0] for i in range(n)]      # ordinary memory: copied
    pin_x = torch.empty(n * c + 3, dtype=torch.float32 if f32_in else torch.uint8).pin_memory()
    rows = pin_x[3:].view(n, c)
    rows.copy_(torch.from_numpy(x.reshape(n, c)))
    pin_y = torch.full((n * k + 2,), 7.0).pin_memory()
    for i in range(n):
        cs.run_host_ptrs(1, [rows[i].data_ptr()], [pin_y[1 + i * k:].data_ptr()])
    got = pin_y.numpy()
    assert np.array_equal(got[1:1 + n * k].reshape(n, k), np.concatenate(want))
    assert got[0] == 7.0 and got[-1] == 7.0
    cs.close()
