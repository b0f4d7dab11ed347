"""Convs that load a tile's activations once for all taps, and convs on groups of pixels: against the CUDA-core kernel, which the
other tests pin to the CPU restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(c, k, r, s, h, w, n, seed, signed=False):
    import torch
    rng = np.random.default_rng(seed)
    wt = rng.integers(-127, 128, (k, c, r, s)).astype(np.int8) if signed else rng.integers(0, 256, (k, c, r, s), dtype=np.uint8)
    bias = rng.integers(-4096, 4097, k).astype(np.int32)
    walpha = rng.uniform(0.001, 0.01, k).astype(np.float32)
    q = dict(ialpha=0.02, walpha=walpha, oalpha=float(np.float32(0.02 * 74 * 0.0055 * 73 * np.sqrt(c * r * s) / (20 if signed else 45))))
    q.update(dict(obits=7, signed=True) if signed else dict(izp=117, ozp=99))
    x = torch.from_numpy(rng.integers(0, 256, (n, h, w, c), dtype=np.uint8)).cuda()
    return wt, bias, x.view(torch.int8) if signed else x, q


# (c, k, kernel (r, s), strides, pads, h, w, n): lines that fill a power of two with their ring and not, maps of one pixel more or
# less than the tiles, planes of a strided window with one and two taps an axis, several channel chunks, an asymmetric window, windows
# of one column with a horizontal stride (the others of those keep a box per tap)
BOXES = [(64, 64, (3, 3), (1, 1), (1, 1), 56, 56, 9), (64, 48, (3, 3), (1, 1), (1, 1), 27, 35, 30), (32, 16, (3, 3), (1, 1), (1, 1), 17, 126, 8),
         (32, 32, (3, 3), (1, 1), (1, 1), 16, 127, 9), (128, 128, (3, 3), (1, 1), (1, 1), 28, 30, 24), (96, 80, (3, 3), (2, 2), (1, 1), 33, 31, 40),
         (16, 256, (3, 3), (1, 1), (0, 0), 10, 9, 60), (48, 96, (5, 3), (1, 2), (2, 1), 30, 29, 20), (160, 32, (2, 4), (2, 1), (1, 3), 21, 23, 30),
         (64, 64, (1, 3), (1, 1), (0, 1), 3, 6, 200), (32, 64, (4, 4), (2, 2), (0, 2), 40, 62, 12),
         (64, 48, (3, 1), (1, 2), (1, 1), 20, 21, 60), (32, 16, (4, 1), (2, 2), (1, 0), 21, 24, 40)]


@pytest.mark.parametrize("shape", BOXES)
@pytest.mark.parametrize("kind", ["plain", "wzp", "signed"])
def test_one_box_for_all_taps(monkeypatch, shape, kind):
    import torch
    from nart_b200 import ops
    c, k, (r, s), st, pad, h, w, n = shape
    wt, bias, x, q = _inputs(c, k, r, s, h, w, n, c + k + h, kind == "signed")
    if kind == "wzp":
        q["wzp"] = 90
    args = dict(in_hw=(h, w), stride=st, pad=pad, relu=kind == "plain", **q)
    want = ops.Conv2d(wt, bias, algo=ops.ALGO_DIRECT, **args)(x)
    monkeypatch.setenv("B200_IGEMM_SMALL", "0")       # launches of any size on the persistent kernel
    monkeypatch.setenv("B200_IGEMM_HALO", "1")
    conv = ops.Conv2d(wt, bias, algo=ops.ALGO_IGEMM, **args)
    for part in (x, x[:1]):
        assert torch.equal(conv(part), want[:part.shape[0]]), conv.describe()
        assert ops.device_status() == 0
    assert len(torch.unique(want)) > 16


def test_the_box_switch_is_read_at_creation(monkeypatch):
    """As the header says of all switches: what the environment holds later changes no plan."""
    import torch
    from nart_b200 import ops
    wt, bias, x, q = _inputs(64, 64, 3, 3, 27, 35, 60, 1)       # a map whose boxes waste too much to be taken by themselves
    args = dict(in_hw=(27, 35), stride=(1, 1), pad=(1, 1), relu=True, **q)
    want = ops.Conv2d(wt, bias, algo=ops.ALGO_DIRECT, **args)(x)
    for value in ("1", "0"):
        plain = ops.Conv2d(wt, bias, **args)
        monkeypatch.setenv("B200_IGEMM_HALO", value)
        switched = ops.Conv2d(wt, bias, **args)
        assert torch.equal(plain(x), want) and "one box" not in plain.describe()
        monkeypatch.delenv("B200_IGEMM_HALO")
        assert torch.equal(switched(x), want) and ("one box" in switched.describe()) == (value == "1")


# (c, k, kernel, strides, pads, h, w): images of four channels and of three, ragged channel counts
GROUPS = [(4, 64, (7, 7), (2, 2), (3, 3), 30, 32), (4, 32, (3, 3), (2, 2), (1, 1), 31, 36), (4, 16, (3, 5), (1, 1), (1, 2), 9, 8), (4, 48, (8, 2), (1, 4), (0, 0), 12, 20),
          (3, 64, (7, 7), (2, 2), (3, 3), 33, 64), (4, 64, (7, 7), (2, 2), (3, 3), 30, 226), (24, 144, (1, 1), (1, 1), (0, 0), 9, 8), (20, 33, (1, 1), (1, 1), (0, 0), 6, 6),
          (24, 40, (3, 3), (1, 1), (1, 1), 11, 14), (8, 48, (3, 3), (1, 1), (1, 1), 10, 12), (8, 33, (1, 5), (1, 1), (0, 2), 7, 6), (8, 64, (3, 3), (2, 2), (1, 1), 15, 18),
          (12, 18, (3, 3), (2, 2), (1, 1), 9, 16), (40, 20, (3, 3), (2, 2), (1, 1), 13, 10), (100, 150, (1, 1), (1, 1), (0, 0), 20, 10)]


@pytest.mark.parametrize("shape", GROUPS)
@pytest.mark.parametrize("size", ["small", "large"])
def test_groups_of_pixels(shape, size):
    """Aligned activations, and a view that only the copy or the lowering takes; both behind one plan, in either order."""
    import torch
    from nart_b200 import ops
    c, k, (r, s), st, pad, h, w = shape
    oh, ow = (h + 2 * pad[0] - r) // st[0] + 1, (w + 2 * pad[1] - s) // st[1] + 1
    n = 1 if size == "small" else -(-148 * 128 * 4 // (oh * ow)) + 1        # four pixels or fewer a group, a tile an SM
    wt, bias, x, q = _inputs(c, k, r, s, h, w, n, c + k + (n > 1))
    args = dict(in_hw=(h, w), stride=st, pad=pad, relu=True, **q)
    want = ops.Conv2d(wt, bias, algo=ops.ALGO_DIRECT, **args)(x)
    shifted = torch.empty(x.numel() + 4, device="cuda", dtype=torch.uint8)[4:].copy_(x.view(-1)).view(x.shape)
    conv, said = ops.Conv2d(wt, bias, **args), []
    for part in (x, shifted, x):
        assert torch.equal(conv(part), want)
        said.append(conv.describe())
    assert ops.device_status() == 0 and conv.algo == ops.ALGO_IGEMM
    if c <= 4:
        groups = size == "large" and w % 4 == 0
        assert ["four-pixel groups" in d for d in said] == [groups, groups and c == 3, groups], said        # (a padded copy is aligned)
    if c == 8 and k % 16 == 0:      # two pixels are the sixteen channels of a box's
        assert ["on groups of pixels" in d for d in said] == [True, False, True], said
    if c == 24 and r == 1:
        assert "groups of pixels" in said[0] and "groups of pixels" not in said[1] and said[2] == said[0]


@pytest.mark.parametrize("pair", ["0", "1"])
def test_pixel_groups_beside_the_cta_pair_switch(monkeypatch, pair):
    """Weights that don't fit beside three ordinary tiles, which is when CTA pairs are considered, but do beside boxes of four-channel
    pixels, which pairs can't read."""
    import torch
    from nart_b200 import ops
    h, w, n = 30, 64, 90
    wt, bias, x, q = _inputs(4, 128, 9, 7, h, w, n, 5)
    args = dict(in_hw=(h, w), stride=(2, 2), pad=(4, 3), relu=True, **q)
    want = ops.Conv2d(wt, bias, algo=ops.ALGO_DIRECT, **args)(x)
    monkeypatch.setenv("B200_IGEMM_CTA_PAIR", pair)
    conv = ops.Conv2d(wt, bias, **args)
    assert torch.equal(conv(x), want) and "four-pixel groups" in conv.describe(), conv.describe()
    assert torch.equal(conv(x[:1]), want[:1]) and ops.device_status() == 0


# (c, k, kernel, pad, h, w): one group more or less than a tile, lines of one group, the largest and smallest widths the rule takes
NARROW = [(32, 16, 1, 0, 28, 28), (64, 64, 1, 0, 13, 26), (48, 17, 1, 0, 6, 10), (16, 96, 1, 0, 9, 14), (256, 32, 1, 0, 7, 4), (96, 32, 1, 0, 16, 8),
          (16, 32, 3, 1, 28, 30), (64, 32, 3, 1, 15, 14), (32, 64, 3, 1, 20, 2), (48, 20, 3, 0, 12, 18), (16, 31, 5, 2, 9, 22)]


@pytest.mark.parametrize("shape", NARROW)
def test_few_output_channels_on_groups_of_pixels(shape):
    """Launches that fill the device and launches that don't, and a view that groups can't read."""
    import torch
    from nart_b200 import ops
    c, k, ks, pad, h, w = shape
    n = -(-148 * 128 * 4 // (h * w)) + 3
    wt, bias, x, q = _inputs(c, k, ks, ks, h, w, n, c + k)
    args = dict(in_hw=(h, w), stride=(1, 1), pad=(pad, pad), relu=False, **q)
    want = ops.Conv2d(wt, bias, algo=ops.ALGO_DIRECT, **args)(x)
    conv = ops.Conv2d(wt, bias, **args)
    assert torch.equal(conv(x), want) and "groups of pixels" in conv.describe(), conv.describe()
    assert torch.equal(conv(x[:2]), want[:2]) and "groups of pixels" not in conv.describe()
    assert torch.equal(conv(x), want) and ops.device_status() == 0


def test_preparation_does_not_grow_with_the_map():
    """All pixels of a 1x1 conv's image are one line of groups: 4 million of them here, of one kind (66 ms when each was looked at)."""
    import time
    from nart_b200 import ops
    wt, bias, _, q = _inputs(16, 16, 1, 1, 8, 8, 1, 2)
    took = []
    for _ in range(5):
        start = time.perf_counter()
        ops.Conv2d(wt, bias, in_hw=(4096, 4096), relu=True, **q)
        took.append(time.perf_counter() - start)
    assert min(took) < 0.015, took


def test_plans_of_maps_of_more_than_two_billion_pixels():
    """Too long a line for groups (its pixels are counted in 31 bits): the plan is made without."""
    from nart_b200 import ops
    wt, bias, _, q = _inputs(16, 16, 1, 1, 8, 8, 1, 2)
    conv = ops.Conv2d(wt, bias, in_hw=(46344, 46344), relu=True, **q)
    assert conv.algo == ops.ALGO_IGEMM


@pytest.mark.parametrize("fused", [False, True])
def test_the_prefetched_weights_are_those_that_are_read(fused):
    """In a case a conv asks for the next one's weights: on groups of pixels from a tile an SM on (twice the columns and twice the
    depth here), and never where that conv has taken over a residual add."""
    from nart_b200.case import Case
    n = 200
    wt, bias, x, q = _inputs(64, 64, 1, 1, 28, 28, n, 6)
    x = x.cpu().numpy().transpose(0, 3, 1, 2).copy()
    cs = Case()
    cs.set_fusion(fused)
    image = cs.input_u8(64, 28, 28)
    a = cs.conv2d(image, wt, bias, **q)
    b = cs.conv2d(a, wt, bias, **q)
    cs.output_u8(cs.eltwise_sum([b, a], (q["oalpha"],) * 2, (q["ozp"],) * 2, 0.05, 120))
    cs.prepare(n)
    for batch, on_groups in ((n, not fused), (1, False), (n, not fused)):
        cs.run_host([x[:batch]], [(np.uint8, (64, 28, 28))])
        first, second = cs.describe()[:2]
        assert ("groups of pixels" in second) == on_groups, second
        assert "prefetches %d bytes" % (64 * 64 * (4 if on_groups else 1)) in first, (batch, first)
    cs.close()


def test_describe_names_what_the_last_run_took():
    """Entry points that never run on groups, after a run that did."""
    import torch
    from nart_b200 import ops
    n = 200
    wt, bias, x, q = _inputs(64, 64, 1, 1, 28, 28, n, 3)
    conv = ops.Conv2d(wt, bias, in_hw=(28, 28), relu=False, **q)
    y = conv(x)
    assert "on groups of pixels" in conv.describe()
    zp = (q["ozp"], 90)
    conv.fuse_residual_add(0, (q["oalpha"], 0.03), zp, 0.05, 120)
    assert torch.equal(conv.run_residual(x, y), ops.add(y, y, (q["oalpha"], 0.03), zp, 0.05, 120))
    assert "groups of pixels" not in conv.describe()
    wt, bias, x, q = _inputs(4, 64, 7, 7, 28, 28, n, 4)
    conv = ops.Conv2d(wt, bias, in_hw=(28, 28), stride=(2, 2), pad=(3, 3), relu=False, **q)
    y = conv(x)
    assert "four-pixel groups" in conv.describe()
    z = torch.empty_like(y)
    assert ops.lib.b200_conv2d_run_static_scratch(conv._h, x.data_ptr(), n, z.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(y, z) and "row-lowered" in conv.describe()


@pytest.mark.parametrize("c,k,ks", [(64, 64, 3), (24, 144, 1), (4, 64, 7)])
def test_run_is_the_first_call_of_a_thread(c, k, ks):
    """A thread that has called nothing of CUDA has no current context."""
    import threading
    import torch
    from nart_b200 import ops
    wt, bias, x, q = _inputs(c, k, ks, ks, 16, 16, 3, c)
    args = dict(in_hw=(16, 16), stride=(1 if c > 4 else 2,) * 2, pad=(ks // 2,) * 2, relu=True, **q)
    want, conv, got = ops.Conv2d(wt, bias, algo=ops.ALGO_DIRECT, **args)(x), ops.Conv2d(wt, bias, **args), []
    torch.cuda.synchronize()
    y = torch.empty_like(want)
    stream = torch.cuda.current_stream().cuda_stream
    t = threading.Thread(target=lambda: got.append(ops.lib.b200_conv2d_run(conv._h, x.data_ptr(), 3, y.data_ptr(), stream)))
    t.start()
    t.join()
    torch.cuda.synchronize()
    assert got == [0] and torch.equal(y, want)
