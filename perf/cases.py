"""The work this framework is used for, as cases whose time can be taken: single convolutions called
op by op, the ops around them, and whole networks through the case runner and the ``art`` interface.

A case is a dict of plain values with one of three kinds:

  conv   one prepared ``ops.Conv2d`` call on NHWC activations that are already on the device
  ops    quantize -> add -> relu -> pool -> dequantize, one ``ops`` call each, on one activation map
  net    one batch through ResNet-18, ResNet-50 or MobileNetV2-1.0, ``via``
           device  ``Case.run_device`` on images already in the input staging buffer, replayed as a graph
           host    ``Case.run_host_ptrs`` on pinned host images, logits back to pinned host memory
           parade  ``art.Parade.run`` on numpy images, the reference's own Python runtime interface

Weights, scales and zero points are synthetic; output scales match the spread of the real values so that the
bytes are distributed over their range, as those of a calibrated network are.  Everything the path returns
is integer arithmetic (the float outputs are one multiplication of an integer), so results are exact.
"""
import math
import os
import tempfile

import numpy as np
import torch

from nart_b200 import art, engine, nets, ops

# What a drawn case may cost at most (bytes moved and integer operations), so that none exceeds the largest
# listed network; the second pair is for what runs on the CUDA cores (grouped convs, ragged channel counts).
MOST_BYTES, MOST_OPS = 400e6, 0.8e12
MOST_BYTES_CUDA, MOST_OPS_CUDA = 200e6, 4e9


def listed():
    conv = dict(kind="conv", ks=3, stride=1, group=1, dtype="u8", wzp=128, relu=True, per_channel=True)
    return [
        # the smallest call: a single 3x3 convolution on one image (latency: launches and host work count)
        dict(conv, name="conv3x3_c64_56_b1", c=64, k=64, h=56, w=56, batch=1),
        # the widest 1x1 expansion of a bottleneck network at serving batch: bound by what it writes
        dict(conv, name="conv1x1_c64_k256_56_b256", c=64, k=256, h=56, w=56, batch=256, ks=1, relu=False),
        # a dense 3x3 contraction at serving batch: bound by the tensor cores
        dict(conv, name="conv3x3_c256_14_b256", c=256, k=256, h=14, w=14, batch=256),
        # weights quantized with a zero point of their own (what a calibrator writes by default), strided
        dict(conv, name="conv3x3s2_wzp_c128_28_b32", c=128, k=128, h=28, w=28, batch=32, stride=2, wzp=117),
        # int8 activations, on a map and a batch that fill no tile
        dict(conv, name="conv3x3_s8_odd_b9", c=64, k=96, h=27, w=35, batch=9, dtype="s8"),
        # a channel count that is no multiple of 16 (MobileNetV2's 24), called op by op
        dict(conv, name="conv1x1_c24_k144_56_b32", c=24, k=144, h=56, w=56, batch=32, ks=1),
        # depthwise
        dict(conv, name="depthwise3x3_c144_56_b64", c=144, k=144, h=56, w=56, batch=64, group=144),
        # the ops around the convolutions on a stem-sized map: memory bound
        dict(name="ops_c64_112_b32", kind="ops", c=64, h=112, w=112, batch=32, method="max"),
        # one image, host to host: the latency of an interactive server
        dict(name="resnet50_b1_host", kind="net", net="resnet50", hw=224, batch=1, via="host"),
        # a case driven through the reference's Python interface
        dict(name="resnet18_b64_parade", kind="net", net="resnet18", hw=224, batch=64, via="parade"),
        # throughput of the two large benchmark networks with the batch resident on the device
        dict(name="mobilenet_v2_b256", kind="net", net="mobilenet_v2", hw=224, batch=256, via="device"),
        dict(name="resnet50_b256", kind="net", net="resnet50", hw=224, batch=256, via="device"),
    ]


# ---- drawing ------------------------------------------------------------------------------------------
def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _out_hw(case):
    p = case["ks"] // 2
    return ((case["h"] + 2 * p - case["ks"]) // case["stride"] + 1, (case["w"] + 2 * p - case["ks"]) // case["stride"] + 1)


def _draw_conv(rng):
    shape = rng.choice(["dense", "dense", "dense", "ragged", "depthwise"])
    if shape == "dense":
        c, k = 16 * _log_int(rng, 1, 32), 16 * _log_int(rng, 1, 64)
    elif shape == "ragged":
        c, k = 4 * _log_int(rng, 1, 50), _log_int(rng, 16, 300)
    else:
        c = k = 16 * _log_int(rng, 2, 60)
    h = _log_int(rng, 7, 112)
    case = dict(kind="conv", c=c, k=k, h=h, w=max(7, h + rng.choice([0, 0, 0, -3, 1, 8])), batch=_log_int(rng, 1, 256),
                ks=3 if shape == "depthwise" else rng.choice([1, 3, 3]), stride=rng.choice([1, 1, 2]),
                group=c if shape == "depthwise" else 1, dtype=rng.choice(["u8", "u8", "u8", "s8"]), wzp=128,
                relu=rng.choice([True, False]), per_channel=rng.choice([True, True, False]))
    if case["dtype"] == "u8" and shape != "depthwise" and rng.random() < 0.25:
        case["wzp"] = rng.randrange(96, 160)
    if shape == "depthwise":
        case["dtype"] = "u8"
    most_bytes, most_ops = (MOST_BYTES, MOST_OPS) if shape == "dense" else (MOST_BYTES_CUDA, MOST_OPS_CUDA)
    while case["batch"] > 1 and (work(case)["bytes"] > most_bytes or work(case)["flops"] > most_ops):
        case["batch"] = (case["batch"] + 1) // 2
    return case


def _draw_ops(rng):
    c = rng.choice([16 * _log_int(rng, 1, 32), 4 * _log_int(rng, 1, 60)])
    h = _log_int(rng, 7, 150)
    case = dict(kind="ops", c=c, h=h, w=max(7, h + rng.choice([0, 0, -2, 1, 5])), batch=_log_int(rng, 1, 128),
                method=rng.choice(["max", "max", "avg"]))
    while case["batch"] > 1 and work(case)["bytes"] > MOST_BYTES:
        case["batch"] = (case["batch"] + 1) // 2
    return case


def _draw_net(rng):
    via = rng.choice(["device", "host", "parade"])
    hw = rng.choice([224, 224, rng.randrange(97, 224)])
    return dict(kind="net", net=rng.choice(["resnet18", "resnet50", "mobilenet_v2"]), hw=hw,
                batch=_log_int(rng, 1, 200 if via == "device" else 64), via=via)


def draw(rng):
    return rng.choice([_draw_conv, _draw_conv, _draw_ops, _draw_net])(rng)


# ---- preparing and running ----------------------------------------------------------------------------
def _scale(x):
    return float(np.float32(x))


def _device_generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _prepare_conv(case, seed):
    rng = np.random.default_rng(seed)
    s8 = case["dtype"] == "s8"
    c, k, ks, group = case["c"], case["k"], case["ks"], case["group"]
    wt = rng.integers(-127, 128, (k, c // group, ks, ks), dtype=np.int16)
    wt = wt.astype(np.int8) if s8 else (wt + 128).astype(np.uint8)
    bias = rng.integers(-4096, 4097, k).astype(np.int32)
    walpha = rng.uniform(0.001, 0.01, k if case["per_channel"] else 1).astype(np.float32)
    taps = c // group * ks * ks
    # activations spread by about 74 around their zero point, weights by about 73: the output scale puts
    # one standard deviation of the result at 45 steps (20 in the 7 bits of the int8 path)
    spread = 0.02 * 74.0 * float(walpha.mean()) * 73.0 * math.sqrt(taps)
    quant = dict(oalpha=_scale(spread / 20.0), obits=7) if s8 else dict(
        izp=int(rng.integers(100, 156)), wzp=case["wzp"], oalpha=_scale(spread / 45.0), ozp=int(rng.integers(60, 180)))
    p = ks // 2
    conv = ops.Conv2d(wt, bias, in_hw=(case["h"], case["w"]), stride=(case["stride"],) * 2, pad=(p, p), group=group,
                      ialpha=0.02, walpha=walpha, relu=case["relu"], signed=s8, **quant)
    x = torch.randint(-127 if s8 else 0, 128 if s8 else 256, (case["batch"], case["h"], case["w"], c),
                      generator=_device_generator(seed), device="cuda", dtype=torch.int8 if s8 else torch.uint8)
    return dict(kind="conv", conv=conv, x=x)


def _prepare_ops(case, seed):
    shape = (case["batch"], case["c"], case["h"], case["w"])
    g = _device_generator(seed)
    rng = np.random.default_rng(seed)
    x = torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)
    res = torch.randint(0, 256, (shape[0], shape[2], shape[3], shape[1]), generator=g, device="cuda", dtype=torch.uint8)
    scales = [_scale(s) for s in rng.uniform(0.01, 0.03, 3)]
    zps = [int(z) for z in rng.integers(90, 166, 3)]
    return dict(kind="ops", x=x, res=res, scales=scales, zps=zps, method=ops.POOL_MAX if case["method"] == "max" else ops.POOL_AVE)


def _spec(case, seed):
    hw = case["hw"]
    if case["net"] == "mobilenet_v2":
        return nets.mobilenet_v2(seed=seed, hw=hw, spread=True)
    return nets.resnet(int(case["net"][6:]), seed=seed, hw=hw, spread=True)


class _DeviceBuffer:
    """A device buffer of the case runner as a torch tensor (``torch.as_tensor`` reads this interface and keeps
    the object, and with it the case that owns the memory, for as long as the tensor lives)."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr=typestr, version=3)


def _prepare_net(case, seed):
    spec, batch, hw = _spec(case, seed), case["batch"], case["hw"]
    images = np.random.default_rng(seed + 1).integers(0, 256, (batch, 3, hw, hw), dtype=np.uint8)
    state = dict(kind="net", via=case["via"], batch=batch)
    if case["via"] == "parade":
        with tempfile.TemporaryDirectory() as d:
            path = os.path.join(d, "engine.bin")
            engine.write_engine(spec, path, batch=batch)
            parade = art.load_parade(path, art.create_context_for_target("b200"))
        inputs, outputs = art.get_empty_io(parade)
        inputs["input"][:] = images
        return dict(state, parade=parade, inputs=inputs, outputs=outputs)
    cs, _ = nets.to_case(spec, batch)
    cs.use_graph(True)
    stream = torch.cuda.Stream()
    state.update(case=cs, stream=stream)
    if case["via"] == "host":
        x = torch.from_numpy(images).pin_memory()
        y = torch.zeros((batch, 1000), dtype=torch.float32).pin_memory()
        return dict(state, x=x, y=y)
    x = torch.as_tensor(_DeviceBuffer(cs, cs.io_device_ptr(False, 0), (batch, 3, hw, hw), "|u1"), device="cuda")
    y = torch.as_tensor(_DeviceBuffer(cs, cs.io_device_ptr(True, 0), (batch, 1000), "<f4"), device="cuda")
    x.copy_(torch.from_numpy(images))
    return dict(state, x=x, y=y)


def prepare(case, seed):
    if case["kind"] == "conv":
        return _prepare_conv(case, seed)
    if case["kind"] == "ops":
        return _prepare_ops(case, seed)
    return _prepare_net(case, seed)


def run(state):
    if state["kind"] == "conv":
        return state["conv"](state["x"])
    if state["kind"] == "ops":
        (a0, a1, a2), (z0, z1, z2) = state["scales"], state["zps"]
        q = ops.quantize(state["x"], a0, z0)
        s = ops.add(q, state["res"], (a0, a1), (z0, z1), a2, z2)
        r = ops.relu(s, a2, z2, a2, z2)
        p = ops.pool(r, state["method"], (3, 3), (1, 1), (2, 2), False, a2, z2, a2, z2)
        return dict(quantized=q, sum=s, relu=r, pooled=p, real=ops.dequantize(p, a2, z2))
    if state["via"] == "parade":
        state["parade"].run(state["inputs"], state["outputs"])
        return state["outputs"]
    if state["via"] == "host":
        state["case"].run_host_ptrs(state["batch"], [state["x"].data_ptr()], [state["y"].data_ptr()], state["stream"].cuda_stream)
        return state["y"]
    state["case"].run_device(state["batch"], state["stream"].cuda_stream)
    return state["y"]


# ---- what a case cannot do without ----------------------------------------------------------------------
# (parameters, multiply-adds per image at 224 x 224) of the three networks, the fully connected layer included
_NETS = {"resnet18": (11.68e6, 1.814e9), "resnet50": (25.5e6, 4.089e9), "mobilenet_v2": (3.47e6, 0.301e9)}


def work(case):
    n = case["batch"]
    if case["kind"] == "conv":
        oh, ow = _out_hw(case)
        cg = case["c"] // case["group"]
        weights = case["k"] * cg * case["ks"] ** 2
        return dict(bytes=n * (case["h"] * case["w"] * case["c"] + oh * ow * case["k"]) + weights + 4 * case["k"],
                    flops=2.0 * n * oh * ow * weights)
    if case["kind"] == "ops":
        oh, ow = (case["h"] - 1) // 2 + 1, (case["w"] - 1) // 2 + 1
        full, pooled = n * case["c"] * case["h"] * case["w"], n * case["c"] * oh * ow
        return dict(bytes=(5 + 3 + 2 + 1) * full + (1 + 5) * pooled, flops=0.0)   # quantize, add, relu, pool, dequantize
    params, macs = _NETS[case["net"]]
    return dict(bytes=n * 3 * case["hw"] ** 2 + params + n * 4000, flops=2.0 * n * macs * (case["hw"] / 224.0) ** 2)


def tolerance(case):
    return "exact"
