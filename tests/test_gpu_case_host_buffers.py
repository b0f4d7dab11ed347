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


def test_a_failed_host_run_leaves_no_buffer_behind():
    """A run that fails on a later input must not leave run_device reading the pinned buffer of an earlier one."""
    from nart_b200.case import Case
    c, h, w = 4, 6, 6
    cs = Case()
    a, b = cs.input_u8(c, h, w), cs.input_u8(c, h, w)
    cs.output_u8(cs.eltwise_sum([a, b], [0.02, 0.02], [0, 0], 0.04, 0))
    cs.prepare(1)
    rng = np.random.default_rng(11)
    x = [torch.from_numpy(rng.integers(0, 256, (1, c, h, w), dtype=np.uint8)).pin_memory() for _ in range(2)]
    (want,) = cs.run_host([t.numpy().copy() for t in x], [(np.uint8, (c, h, w))])       # fills the staging buffers
    with pytest.raises(Exception, match="input 1 is NULL"):
        cs.run_host_ptrs(1, [x[0].data_ptr(), None], [x[1].data_ptr()])
    x[0].zero_()
    cs.run_device(1)
    torch.cuda.synchronize()
    from nart_b200._lib import check, lib
    got = np.empty_like(want)
    check(lib.b200_memcpy_d2h(got.ctypes.data, cs.io_device_ptr(True, 0), got.nbytes, None))
    torch.cuda.synchronize()
    assert np.array_equal(got, want)
    cs.close()
