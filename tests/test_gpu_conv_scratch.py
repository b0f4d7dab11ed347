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


def _direct(c, k, hw):
    from nart_b200 import ops
    return _plan(c, k, hw, algo=ops.ALGO_DIRECT)


# (channels, output channels, map, batch): 24 -> 32 channels; an image of 3 channels, which is lowered as well
SHARED = [(24, 144, 56, 16), (3, 32, 56, 16)]


@pytest.mark.parametrize("c,k,hw,n", SHARED)
def test_one_plan_on_several_streams(c, k, hw, n):
    plan = _plan(c, k, hw)
    xs = [torch.randint(0, 256, (n + i, hw, hw, c), device="cuda", dtype=torch.uint8) for i in range(4)]
    want = [_direct(c, k, hw)(x) for x in xs]
    streams = [torch.cuda.Stream() for _ in xs]
    plan(xs[-1])
    torch.cuda.synchronize()
    torch.cuda._sleep(20_000_000)       # all is queued before any of it runs
    for st in streams:
        st.wait_stream(torch.cuda.current_stream())
    got = []
    for _ in range(25):
        for x, st in zip(xs, streams):
            with torch.cuda.stream(st):
                got.append(plan(x))
    torch.cuda.synchronize()
    for i, y in enumerate(got):
        assert torch.equal(y, want[i % len(xs)]), i


@pytest.mark.parametrize("c,k,hw,n", SHARED)
def test_one_plan_in_several_threads(c, k, hw, n):
    import threading
    plan = _plan(c, k, hw)
    xs = [torch.randint(0, 256, (n, hw, hw, c), device="cuda", dtype=torch.uint8) for _ in range(4)]
    want = [_direct(c, k, hw)(x) for x in xs]
    torch.cuda.synchronize()
    bad = []

    def work(i, stream):
        with torch.cuda.stream(stream):
            got = [plan(xs[i]) for _ in range(40)]
            torch.cuda.current_stream().synchronize()
        bad.extend(i for y in got if not torch.equal(y, want[i]))

    shared = torch.cuda.Stream()        # two threads on one stream, two on their own
    threads = [threading.Thread(target=work, args=(i, shared if i < 2 else torch.cuda.Stream())) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("c,k,hw,n", SHARED)
def test_first_run_under_capture_and_replays_beside_growth(c, k, hw, n):
    plan, direct = _plan(c, k, hw), _direct(c, k, hw)
    x = torch.randint(0, 256, (2, hw, hw, c), device="cuda", dtype=torch.uint8)
    big = torch.randint(0, 256, (3 * n, hw, hw, c), device="cuda", dtype=torch.uint8)
    want_big = direct(big)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = plan(x)
        z = plan(x[1:])
    for seed in range(3):
        x.random_(0, 256)
        want = direct(x)
        torch.cuda.synchronize()
        eager = [plan(big[:n * (seed + 1)]) for _ in range(3)]      # grows the plan's own buffer
        g.replay()
        eager += [plan(big[:n * (seed + 1)]) for _ in range(3)]
        torch.cuda.synchronize()
        assert torch.equal(y, want) and torch.equal(z, want[1:])
        assert all(torch.equal(e, want_big[:n * (seed + 1)]) for e in eager)


def test_captures_behind_a_large_run_of_a_four_channel_image():
    """A run on groups of pixels uses no scratch, but sizes it: smaller batches and views that groups can't read are captured behind it
    without an allocation, and the graph's scratch stays where it is."""
    c, k, hw, n = 4, 32, 56, 64
    plan, direct = _plan(c, k, hw), _direct(c, k, hw)
    big = torch.randint(0, 256, (n, hw, hw, c), device="cuda", dtype=torch.uint8)
    shifted = torch.empty(big.numel() + 4, device="cuda", dtype=torch.uint8)[4:].view(big.shape).copy_(big)
    want = direct(big)
    assert torch.equal(plan(big), want) and "four-pixel groups" in plan.describe()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        one = plan(big[:1])
        views = plan(shifted)
    for m in (3, 24, n):            # (none of them moves the scratch)
        assert torch.equal(plan(big[:m]), want[:m]) and torch.equal(plan(shifted[:m]), want[:m])
        one.zero_(), views.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(one, want[:1]) and torch.equal(views, want)


def test_a_large_run_without_memory_for_rows_leaves_those_there_are():
    """A run on groups needs no rows itself: it goes on, and what an earlier graph reads stays."""
    from nart_b200._lib import lib
    c, k, hw, n = 4, 32, 56, 2000           # 200 MB of rows
    plan, direct = _plan(c, k, hw), _direct(c, k, hw)
    x = torch.randint(0, 256, (n, hw, hw, c), device="cuda", dtype=torch.uint8)
    y = torch.zeros((n, hw, hw, k), device="cuda", dtype=torch.uint8)
    want = direct(x)
    assert torch.equal(plan(x[:20]), want[:20]) and "row-lowered" in plan.describe()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        one = plan(x[:1])
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    filler = torch.empty(free - (120 << 20), device="cuda", dtype=torch.uint8)
    for _ in range(2):
        y.zero_()
        assert lib.b200_conv2d_run(plan._h, x.data_ptr(), n, y.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        assert "four-pixel groups" in plan.describe()
    del filler
    torch.cuda.empty_cache()
    one.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want) and torch.equal(one, want[:1])
    assert torch.equal(plan(x[:20]), want[:20])


def test_first_run_of_a_process_under_capture():
    """Nothing that a capture forbids is left to the first run."""
    import os
    import subprocess
    import sys
    code = """
import torch
from tests.test_gpu_conv_scratch import _direct, _plan
plan = _plan(24, 144, 14)
x = torch.randint(0, 256, (2, 14, 14, 24), device="cuda", dtype=torch.uint8)
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    y = plan(x)
g.replay()
torch.cuda.synchronize()
assert torch.equal(y, _direct(24, 144, 14)(x))
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    res = subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, PYTHONPATH=root), capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]


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


def test_case_counts_the_copy_into_the_padded_tensor(port):
    from nart_b200.case import Case
    rng = np.random.default_rng(5)
    x = rng.integers(0, 256, (2, 20, 9, 9), dtype=np.uint8)
    wt = rng.integers(0, 256, (32, 20, 3, 3), dtype=np.uint8)
    q = dict(ialpha=0.02, izp=120, walpha=np.float32([0.005]), oalpha=0.5, ozp=99)
    cs = Case()
    cs.output_u8(cs.conv2d(cs.input_u8(20, 9, 9), wt, None, pad=(1, 1), **q))
    cs.prepare(2)
    assert cs.launch_count() == 4       # input layout, padding, convolution, output layout
    (got,) = cs.run_host([x], [(np.uint8, (32, 9, 9))])
    cs.close()
    assert np.array_equal(got, port.conv2d_u8(x, wt, np.zeros(32, np.int32), (1, 1), (1, 1), 1, 0.02, 120, q["walpha"], 128, 0.5, 99))


def test_case_keeps_no_copy_for_a_conv_that_runs_on_groups():
    """24 channels on pairs of pixels at every batch: the case holds its tensors and staging buffers, and no padded tensor beside them."""
    from nart_b200.case import Case
    rng = np.random.default_rng(6)
    n, hw = 200, 112
    wt = rng.integers(0, 256, (32, 24, 1, 1), dtype=np.uint8)
    cs = Case()
    cs.output_u8(cs.conv2d(cs.input_u8(24, hw, hw), wt, None, ialpha=0.02, izp=120, walpha=np.float32([0.005]), oalpha=0.5, ozp=99))
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    cs.prepare(n)
    held = before - torch.cuda.mem_get_info()[0]
    pixels = n * hw * hw
    assert held < 2 * pixels * (24 + 32) + (32 << 20), held         # (with the copy 32 bytes a pixel more, 80 MB)
    assert cs.launch_count() == 3
    x = rng.integers(0, 256, (n, 24, hw, hw), dtype=np.uint8)
    (got,) = cs.run_host([x], [(np.uint8, (32, hw, hw))])
    cs.close()
    from nart_b200 import ops
    plan = ops.Conv2d(wt, None, in_hw=(hw, hw), algo=ops.ALGO_DIRECT, ialpha=0.02, izp=120, walpha=np.float32([0.005]), oalpha=0.5, ozp=99)
    want = plan(torch.from_numpy(x).cuda().permute(0, 2, 3, 1).contiguous())
    assert torch.equal(torch.from_numpy(got).cuda().view(n, 32, hw, hw).permute(0, 2, 3, 1), want)
