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


def _staged_output(cs, want):
    from nart_b200._lib import check, lib
    got = np.empty_like(want)
    check(lib.b200_memcpy_d2h(got.ctypes.data, cs.io_device_ptr(True, 0), got.nbytes, None))
    torch.cuda.synchronize()
    return got


@pytest.mark.parametrize("ask_first", [False, True])
def test_resident_run_after_host_runs(ask_first):
    """run_device works on what the host runs before it brought to the device, image by image, and the staging buffers hold
    what they copied in and out -- whether or not the host runs used the caller's pinned buffers in their place."""
    from nart_b200.case import Case
    c, h, w, n = 3, 6, 5, 4
    rng = np.random.default_rng(12)
    cs = Case()
    t = cs.input_u8(c, h, w)
    t = cs.conv2d(t, rng.integers(0, 256, (32, c, 3, 3), dtype=np.uint8), None, pad=(1, 1), ialpha=0.02, izp=120, walpha=0.005,
                  oalpha=0.1, ozp=111)
    cs.output_f32(t, 0.1, 111)
    cs.prepare(n)
    a, b = (rng.integers(0, 256, (n, c, h, w), dtype=np.uint8) for _ in range(2))
    (want_a,), (want_b,) = (cs.run_host([v], [(np.float32, (32, h, w))]) for v in (a, b))
    if ask_first:
        cs.io_device_ptr(False, 0)
    pin_a, pin_b = (torch.from_numpy(v).pin_memory() for v in (a, b))
    y = torch.zeros((n, 32, h, w)).pin_memory()
    cs.run_host_ptrs(n, [pin_a.data_ptr()], [y.data_ptr()])
    assert np.array_equal(y.numpy(), want_a)
    cs.run_host_ptrs(2, [pin_b.data_ptr()], [y.data_ptr()])
    mixed = np.concatenate([want_b[:2], want_a[2:]])
    assert np.array_equal(y.numpy(), mixed)
    pin_a.zero_(), pin_b.zero_()
    cs.run_device(n)
    torch.cuda.synchronize()
    assert np.array_equal(_staged_output(cs, mixed), mixed)
    # and a caller who has the staging buffer's address finds a host run's results and inputs there
    pin_b.copy_(torch.from_numpy(b))
    cs.run_host_ptrs(n, [pin_b.data_ptr()], [y.data_ptr()])
    assert np.array_equal(_staged_output(cs, want_b), want_b)
    cs.run_device(n)
    torch.cuda.synchronize()
    assert np.array_equal(_staged_output(cs, want_b), want_b)
    cs.close()


def test_staging_address_asked_for_after_a_host_run():
    """The first look at the staging buffers comes behind a host run on pinned buffers: both hold its data."""
    from nart_b200._lib import check, lib
    cs, c = _logits_case(10, False)
    rng = np.random.default_rng(4)
    x = rng.integers(0, 256, (2, c, 1, 1), dtype=np.uint8)
    (want,) = cs.run_host([x], [(np.float32, (10,))])
    cs.run_host([np.zeros_like(x)], [(np.float32, (10,))])
    pin_x, pin_y = torch.from_numpy(x).pin_memory(), torch.zeros((2, 10)).pin_memory()
    cs.run_host_ptrs(2, [pin_x.data_ptr()], [pin_y.data_ptr()])
    assert np.array_equal(_staged_output(cs, want), want)
    got = np.empty_like(x)
    check(lib.b200_memcpy_d2h(got.ctypes.data, cs.io_device_ptr(False, 0), got.nbytes, None))
    torch.cuda.synchronize()
    assert np.array_equal(got, x)
    cs.close()


def test_parade_forward_after_run(tmp_path):
    """Parade.forward runs on the data that Parade.run brought to the device."""
    import os

    from nart_b200 import art, engine, nets
    spec = nets.resnet(18, seed=23, hw=64, width_div=4, spread=True, num_classes=10)
    path = os.path.join(tmp_path, "engine.bin")
    engine.write_engine(spec, path, batch=2)
    parade = art.load_parade(path, art.create_context_for_target("b200"))
    inputs, outputs = art.get_empty_io(parade)
    (iname,), (oname,) = parade.get_input_names(), parade.get_output_names()
    for seed in (5, 6):
        inputs[iname][:] = np.random.default_rng(seed).integers(0, 256, inputs[iname].shape, dtype=np.uint8)
        parade.run(inputs, outputs)
        want = outputs[oname].copy()
        outputs[oname].fill(0)
        parade.forward()
    assert np.array_equal(_staged_output(parade._case, want), want)
    parade.close()


def test_parade_run_into_arrays_of_any_kind(tmp_path):
    """Byte order, strides and alignment of the output arrays are the caller's: values are assigned, not bytes."""
    import os

    from nart_b200 import art, engine, nets
    spec = nets.resnet(18, seed=23, hw=64, width_div=4, spread=True, num_classes=10)
    path = os.path.join(tmp_path, "engine.bin")
    engine.write_engine(spec, path, batch=2)
    parade = art.load_parade(path, art.create_context_for_target("b200"))
    inputs, outputs = art.get_empty_io(parade)
    (iname,), (oname,) = parade.get_input_names(), parade.get_output_names()
    inputs[iname][:] = np.random.default_rng(5).integers(0, 256, inputs[iname].shape, dtype=np.uint8)
    parade.run(inputs, outputs)
    want, shape = outputs[oname].copy(), outputs[oname].shape
    assert len(np.unique(want)) > 3
    kinds = [np.zeros(shape, ">f4"), np.zeros((2 * shape[0],) + shape[1:], np.float32)[::2], np.zeros(shape[:1] + (12, 1, 1), ">f4")[:, 1:11],
             np.zeros(4 * want.size + 1, np.uint8)[1:].view(np.float32).reshape(shape)]
    for y in kinds:
        parade.run(inputs, {oname: y})
        assert np.array_equal(y, want)
    parade.close()


class _Buffer:
    """Device memory as a torch tensor."""

    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr=typestr, version=3)


@pytest.mark.parametrize("net,hw,batch", [("resnet18", 224, 96), ("mobilenet_v2", 224, 65), ("resnet50", 176, 134)])
@pytest.mark.parametrize("pinned", [True, False])
def test_images_that_are_copied_in_two_parts(net, hw, batch, pinned):
    """Graph mode, batches whose first part has 45 us of work and more: eager, captured and replayed runs with other images each time,
    against runs on images that are on the device already; smaller batches of the same case, and a run without a graph, in between."""
    from nart_b200 import nets
    spec = nets.mobilenet_v2(seed=3, hw=hw, spread=True) if net == "mobilenet_v2" else nets.resnet(int(net[6:]), seed=3, hw=hw, spread=True, width_div=2)
    cs, _ = nets.to_case(spec, batch)
    ref, _ = nets.to_case(spec, batch)
    cs.use_graph(True)
    stream = torch.cuda.Stream()
    x_dev = torch.as_tensor(_Buffer(ref.io_device_ptr(False, 0), (batch, 3, hw, hw), "|u1"), device="cuda")
    y_dev = torch.as_tensor(_Buffer(ref.io_device_ptr(True, 0), (batch, 1000), "<f4"), device="cuda")
    x, y = torch.empty((batch, 3, hw, hw), dtype=torch.uint8), torch.empty((batch, 1000), dtype=torch.float32)
    if pinned:
        x, y = x.pin_memory(), y.pin_memory()
    for i, n in enumerate([batch, batch, batch, 7, batch, 32, 32, batch, batch]):
        x.random_(0, 256)
        cs.use_graph(i != 4)
        cs.run_host_ptrs(n, [x.data_ptr()], [y.data_ptr()], stream.cuda_stream)
        x_dev.copy_(x)
        torch.cuda.synchronize()
        ref.run_device(n, 0)
        torch.cuda.synchronize()
        assert torch.equal(y[:n], y_dev[:n].cpu()), i
        assert ("in parts of %d and" % (n // 32 * 16) in cs.describe()[-1]) == (n == batch and i != 4), (i, cs.describe()[-1])
    cs.close()
    ref.close()


def _two_branches(batch):
    """A float and a byte image, each through a stem and a 3x3 conv, and their sum: bytes and, pooled, floats."""
    from nart_b200.case import Case
    rng = np.random.default_rng(8)
    q = dict(ialpha=0.02, izp=117, oalpha=0.4, ozp=99, walpha=np.float32([0.004]))
    cs = Case()
    ends = []
    for image in (cs.input_f32(3, 96, 128, 0.02, 117), cs.input_u8(4, 96, 128)):
        stem = cs.conv2d(image, rng.integers(0, 256, (64, cs.dims(image)[0], 7, 7), dtype=np.uint8), None, stride=(2, 2), pad=(3, 3), **q)
        ends.append(cs.conv2d(stem, rng.integers(0, 256, (64, 64, 3, 3), dtype=np.uint8), None, pad=(1, 1), **dict(q, ialpha=0.4, izp=99, oalpha=11.0)))
    total = cs.eltwise_sum(ends, (11.0, 11.0), (99, 99), 14.0, 120)
    pooled = cs.pool(total, 0, (8, 8), (0, 0), (8, 8), False, 14.0, 120, 14.0, 120)
    cs.output_u8(pooled)
    cs.output_f32(total, 14.0, 120)
    cs.prepare(batch)
    return cs


def test_two_inputs_that_are_copied_in_two_parts():
    batch = 187
    cs, ref = _two_branches(batch), _two_branches(batch)
    cs.use_graph(True)
    stream = torch.cuda.Stream()
    shapes = [((batch, 3, 96, 128), "<f4"), ((batch, 4, 96, 128), "|u1"), ((batch, 64, 6, 8), "|u1"), ((batch, 64, 48, 64), "<f4")]
    dev = [torch.as_tensor(_Buffer(ref.io_device_ptr(i > 1, i % 2), *shapes[i]), device="cuda") for i in range(4)]
    host = [torch.empty(s, dtype=torch.uint8 if t == "|u1" else torch.float32).pin_memory() for s, t in shapes]
    for i, n in enumerate([batch, batch, batch, 40, batch]):
        host[0].normal_(0, 1.5)
        host[1].random_(0, 256)
        cs.run_host_ptrs(n, [h.data_ptr() for h in host[:2]], [h.data_ptr() for h in host[2:]], stream.cuda_stream)
        for d, h in zip(dev, host[:2]):
            d.copy_(h)
        torch.cuda.synchronize()
        ref.run_device(n, 0)
        torch.cuda.synchronize()
        for d, h in zip(dev[2:], host[2:]):
            assert torch.equal(h[:n], d[:n].cpu()) and len(torch.unique(d[:n])) > 8, i
        assert ("in parts of 80 and 107" in cs.describe()[-1]) == (n == batch), (i, cs.describe()[-1])
    cs.close()
    ref.close()
