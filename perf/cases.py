"""Workloads of the int8 convolution path: what users of the library have it do, through its public calls.

Twelve listed cases and a generator of further ones (`draw`) over the same ranges:

* single quantized layers (`ConvInt8.forward` on device buffers): 1x1, 3x3 and depthwise 3x3 / 5x5 convolutions from one image
  to batches of 128, fp32 or int8 in and out, every activation and both rounding rules;
* the ShuffleNetV2-1.0x backbone: one image at a time from host memory (`Net.forward`), a serving loop that replays a
  captured forward on device buffers (`Net.capture`), and large batches from pinned host memory (`Net.forward_raw`);
* the NanoDet-Plus detector: one camera frame in, its boxes out (`Net.forward_rows`; the shipped 1.5x graph at 416x416), and
  batches whose captured forward is followed by the decode of every image (`ott_nanodet_detect`).

A case is a dict of plain values; `prepare(case, seed)` makes its inputs (from the seed) and the layer or Net that runs it,
`run(state)` makes one pass. Model weights do not depend on the seed: a program keeps one model and feeds it new images.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from tensor_b200 import (ACT_LRELU, ACT_NONE, ACT_RELU, ACT_RELU6, F32_NCHW, ROUND_ADD_HALF_TRUNC, ROUND_HALF_AWAY, S8_NHWC,
                         ConvInt8, Context, Net, graphs, nhwc_channels)

ACTS = {"none": ACT_NONE, "relu": ACT_RELU, "lrelu": ACT_LRELU, "relu6": ACT_RELU6}
ROUNDINGS = {"packed": ROUND_ADD_HALF_TRUNC, "away": ROUND_HALF_AWAY}
WIDTHS = {"1.0x": dict(neck=96, stage_channels=(116, 232, 464)), "1.5x": dict(neck=128, stage_channels=(176, 352, 704))}
CLASSES, REG_BINS = 80, 8
PROB_THRESHOLD, NMS_THRESHOLD, MAX_DETECTIONS = 0.4, 0.5, 256


def _layer(name, cin, cout, k, stride, n, h, w, src, dst, act, depthwise=False, rounding="packed"):
    return dict(name=name, kind="layer", cin=cin, cout=cout, k=k, stride=stride, depthwise=depthwise, n=n, h=h, w=w, src=src, dst=dst, act=act,
                rounding=rounding)


def listed():
    return [
        # one 3x3 layer on one image, fp32 on both sides: a single layer of a reference Net moved to the GPU. Launch latency.
        _layer("conv3x3_one_image", 64, 64, 3, 1, 1, 56, 56, "f32", "f32", "none"),
        # a ShuffleNetV2 stage-3 width, which is no multiple of 32, on an odd map, with the scalar / aarch64 rounding rule
        _layer("pw116_odd_map_away", 116, 116, 1, 1, 40, 19, 27, "s8", "s8", "relu", rounding="away"),
        # pointwise sweep of the benchmark configurations, fp32 input quantized on the way in
        _layer("pw256_512_f32_in", 256, 512, 1, 1, 128, 28, 28, "f32", "s8", "relu6"),
        # the widest layer of that sweep, fed by a requantizing producer: the most arithmetic in one launch
        _layer("pw512_1024_s8", 512, 1024, 1, 1, 128, 56, 56, "s8", "s8", "relu6"),
        # a down-sampling 3x3 layer on an odd map, int8 in, fp32 out
        _layer("conv3x3_s2_odd_map", 64, 128, 3, 2, 32, 75, 75, "s8", "f32", "lrelu"),
        # depthwise configuration: fp32 in, int8 out
        _layer("dw3x3_256_f32_in", 256, 256, 3, 1, 64, 56, 56, "f32", "s8", "relu", depthwise=True),
        # the 5x5 depthwise layer of the detector's heads, between two int8 layers
        _layer("dw5x5_96_s8", 96, 96, 5, 1, 32, 40, 40, "s8", "s8", "lrelu", depthwise=True),
        # classification of one image: host array in, feature map out
        dict(name="backbone_one_image", kind="backbone", mode="host", n=1, h=320, w=320),
        # a serving loop on device buffers at the benchmark's batch
        dict(name="backbone_graph_256", kind="backbone", mode="graph", n=256, h=320, w=320),
        # a host batch that is no multiple of the 64-image chunks the library cuts it into, from pinned memory
        dict(name="backbone_pinned_150", kind="backbone", mode="pinned", n=150, h=320, w=320),
        # one camera frame through the detector the reference ships, boxes out
        dict(name="detector_one_frame", kind="detector", mode="host", width="1.5x", n=1, h=416, w=416),
        # a batch of frames on device buffers, heads by a captured forward and every image decoded
        dict(name="detector_graph_32", kind="detector", mode="graph", width="1.0x", n=32, h=320, w=320),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5))))))


def draw(rng):
    kind = rng.choice(("pointwise", "conv3x3", "depthwise", "backbone", "detector"))
    if kind in ("pointwise", "conv3x3", "depthwise"):
        src, dst = rng.choice(("f32", "s8", "s8")), rng.choice(("f32", "s8", "s8"))
        act, rounding = rng.choice(tuple(ACTS)), rng.choice(("packed", "packed", "packed", "away"))
        n, h, w = _log_int(rng, 1, 128), _log_int(rng, 7, 80), _log_int(rng, 7, 80)
        if kind == "depthwise":
            c = _log_int(rng, 24, 512)
            case = _layer("", c, c, rng.choice((3, 3, 5)), rng.choice((1, 1, 2)), n, h, w, src, dst, act, True, rounding)
        else:
            k = 1 if kind == "pointwise" else 3
            top = 1024 if k == 1 else 256
            case = _layer("", _log_int(rng, 24, top), _log_int(rng, 24, top), k, rng.choice((1, 1, 2)) if k == 3 else 1, n, h, w, src, dst, act, False,
                          rounding)
        while work(case)["bytes"] > 6e8 or work(case)["flops"] > 4e11:
            case["n"] //= 2
    elif kind == "backbone":
        mode = rng.choice(("host", "graph", "graph", "pinned"))
        lo, hi = {"host": (1, 8), "graph": (1, 256), "pinned": (16, 200)}[mode]
        case = dict(kind=kind, mode=mode, n=_log_int(rng, lo, hi), h=rng.randint(160, 416), w=rng.randint(160, 416))
        case["n"] = max(1, min(case["n"], 200 * 320 * 320 // (case["h"] * case["w"])))
    else:
        mode = rng.choice(("host", "graph"))
        case = dict(kind=kind, mode=mode, width=rng.choice(("1.0x", "1.5x")), n=1 if mode == "host" else _log_int(rng, 1, 64), h=32 * rng.randint(7, 15),
                    w=32 * rng.randint(7, 15))
        case["n"] = max(1, min(case["n"], 64 * 320 * 320 // (case["h"] * case["w"])))
    case.pop("name", None)
    return case


# ---- single layers ----------------------------------------------------------------------------------------------------------

def _out_hw(case):
    return tuple((v + 2 * (case["k"] // 2) - case["k"]) // case["stride"] + 1 for v in (case["h"], case["w"]))


@functools.lru_cache(maxsize=None)
def _context():
    return Context(0)  # one per GPU and program: its stream and its allocator


class _Handle:
    """Closes a library object when the last state or output that uses it is gone."""

    def __init__(self, *objects):
        self.objects = objects

    def __del__(self):
        for o in self.objects:
            o.close()


def _quantized(rng, shape, std):
    wf = rng.normal(0.0, std, size=shape).astype(np.float32)
    scales = (np.float32(127.0) / np.abs(wf).reshape(shape[0], -1).max(axis=1)).astype(np.float32)
    return np.clip(np.rint(wf * scales[:, None, None, None]), -127, 127).astype(np.int8), scales


def _prepare_layer(case, seed):
    cin, cout, k, n, h, w = (case[i] for i in ("cin", "cout", "k", "n", "h", "w"))
    dw = case["depthwise"]
    rng = np.random.default_rng(0x0771E5)
    std = 0.1 if dw else 0.05
    weight, w_scales = _quantized(rng, (cout, 1 if dw else cin, k, k), std)
    top = 4.0 * std * math.sqrt((1 if dw else cin) * k * k / 3.0)  # activations are uniform [-1, 1]: four sigma of the sums
    if case["act"] == "relu6":
        top = min(top, 6.0)
    scales = cin if dw else 1
    layer = ConvInt8(_context(), cin=cin, cout=cout, kh=k, kw=k, sh=case["stride"], sw=case["stride"], ph=k // 2, pw=k // 2, groups=cin if dw else 1,
                     int8_scale_term=101 if case["dst"] == "s8" else 1, act_type=ACTS[case["act"]], act_param0=0.1 if case["act"] == "lrelu" else 0.0,
                     rounding=ROUNDINGS[case["rounding"]], weight=weight, bias=rng.normal(0.0, 0.01, size=cout).astype(np.float32), w_scales=w_scales,
                     in_scales=np.full(scales, 127.0, np.float32), out_scales=np.full(scales, 127.0 / top, np.float32) if case["dst"] == "s8" else None)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["src"] == "f32":
        x = torch.rand((n, cin, h, w), generator=gen, device="cuda") * 2 - 1
    else:
        x = torch.zeros((n, h, w, nhwc_channels(cin)), dtype=torch.int8, device="cuda")
        x[..., :cin] = torch.randint(-127, 128, (n, h, w, cin), generator=gen, device="cuda", dtype=torch.int8)
    oh, ow = _out_hw(case)
    y = (torch.zeros((n, oh, ow, nhwc_channels(cout)), dtype=torch.int8, device="cuda") if case["dst"] == "s8" else
         torch.zeros((n, cout, oh, ow), device="cuda"))
    return dict(kind="layer", layer=layer, handle=_Handle(layer), x=x, src=F32_NCHW if case["src"] == "f32" else S8_NHWC, n=n, h=h, w=w, y=y,
                dst=S8_NHWC if case["dst"] == "s8" else F32_NCHW)


# ---- whole graphs -----------------------------------------------------------------------------------------------------------

def _layers(case, h, w, batch=1):
    if case["kind"] == "backbone":
        return graphs.shufflenetv2_layers(h, w, batch=batch)
    return graphs.nanodet_plus_layers(h, w, batch=batch, detect=case["mode"] == "host", **WIDTHS[case["width"]])


def _scale_for(x):
    """127 / max|x|, rounded down to an eighth of an octave, so that it does not hang on the last bits of the calibration."""
    return np.float32(2.0 ** (math.floor(8 * math.log2(127.0 / max(float(x.abs().max()), 1e-6))) / 8))


@functools.lru_cache(maxsize=None)
def _model(kind, width):
    """Weights and calibrated activation scales by layer name: one float pass of a small image through the graph, as a
    quantization tool makes it. The heads are scaled and biased like a trained detector's: a few per cent of the cells pass the
    threshold."""
    layers = _layers(dict(kind=kind, mode="graph", width=width), 128, 128)
    params, geometry, blobs, int8_scale = graphs.make_params(layers), graphs.conv_geometry(layers), {}, {}
    F = torch.nn.functional
    for l in layers:
        ins = [blobs[s.strip()] for s in str(l.get("input", "")).split(",") if s.strip()]
        t, name = l["type"], l["name"]
        if t == "Input":
            y = torch.rand((1, 3, 128, 128), generator=torch.Generator().manual_seed(0x0771E5))
        elif t == "Convolution":
            g, p = geometry[name], params[name]
            scales = g["groups"] if g["groups"] > 1 else 1
            p["in_scales"] = np.full(scales, int8_scale.get(g["input"]) or _scale_for(ins[0]), np.float32)
            weight = torch.from_numpy(p["weight"].astype(np.float32) / p["w_scales"][:, None, None, None])
            y = F.conv2d(ins[0], weight, torch.from_numpy(p["bias"]), g["stride"], g["pad"], 1, g["groups"])
            y = {0: lambda v: v, 1: F.relu, 2: lambda v: F.leaky_relu(v, 0.1), 3: lambda v: v.clamp(0, 6)}[g["act"]](y)
            if g["term"] > 100:
                int8_scale[name] = _scale_for(y)
                p["out_scales"] = np.full(scales, int8_scale[name], np.float32)
            if name in graphs.NANODET_OUTPUTS:
                gain = 2.0 ** round(-math.log2(float(y.std())))  # logits spread over a few units, as a trained head's do
                p["w_scales"], p["bias"], y = p["w_scales"] / np.float32(gain), p["bias"] * np.float32(gain), y * gain
                best = y[0, :CLASSES].amax(dim=0).flatten()
                p["bias"][:CLASSES] -= np.float32(round(float(best.mean() + 2 * best.std(correction=0)) - math.log(PROB_THRESHOLD / (1 - PROB_THRESHOLD)), 2))
        elif t == "MaxPool":
            y = F.max_pool2d(ins[0], 3, 2, 1)
        elif t == "Concat":
            y = torch.cat(ins, dim=1)
        elif t == "Crop":
            y = ins[0][:, int(l["start"]):int(l["end"])]
        elif t == "ChannelShuffle":
            y = F.channel_shuffle(ins[0], int(l["groups"]))
        elif t == "ShortCut":
            y = ins[0] + ins[1]
        else:
            y = F.interpolate(ins[0], scale_factor=float(l["stride"]), mode="bilinear", align_corners=False)
        blobs[l["output"]] = y
    return params


class _DeviceArray:
    """A device tensor of the library as torch sees it; keeps its owner alive."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=tuple(shape), typestr="<f4", version=3)


def _prepare_net(case, seed):
    n, h, w = case["n"], case["h"], case["w"]
    net = Net(0)
    for l in _layers(case, h, w, n):
        net.add_layer(**l)
    net.compile()
    for name, p in _model(case["kind"], case.get("width", "1.0x")).items():
        net.set_conv_params(name, p["weight"], p["bias"], p["w_scales"], p["in_scales"], p["out_scales"])
    state = dict(kind=case["kind"], mode=case["mode"], net=net, shape=(n, 3, h, w))
    if case["mode"] == "host":
        state["handle"] = _Handle(net)
        state["x"] = np.random.default_rng(seed).random((n, 3, h, w), dtype=np.float32)
        state["cells"] = sum(math.prod(net.blob_shape(b)[2:]) for b in graphs.NANODET_OUTPUTS) if case["kind"] == "detector" else 0
        return state
    x = torch.rand((n, 3, h, w), generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")
    if case["mode"] == "pinned":
        state["handle"] = _Handle(net)
        state["x"] = torch.empty(x.shape, pin_memory=True).copy_(x)
        state["y"] = torch.zeros((n,) + net.blob_shape("conv5")[1:], pin_memory=True)
        return state
    torch.cuda.synchronize()  # the library's stream reads x from here on
    outputs = ["conv5"] if case["kind"] == "backbone" else list(graphs.NANODET_OUTPUTS)
    graph = net.capture("data", C.c_void_p(x.data_ptr()), (n, 3, h, w), outputs)
    owner = _Handle(graph, net)
    buffers = [graph.output(i) for i in range(len(outputs))]
    state.update(handle=owner, x=x, graph=graph, outputs=[torch.as_tensor(_DeviceArray(p, s, owner), device="cuda") for p, s in buffers])
    if case["kind"] == "detector":
        state["ctx"] = net.context()
        state["heads"] = (C.c_void_p * len(buffers))(*[p for p, _ in buffers])
        state["grid_h"], state["grid_w"] = (np.array([s[i] for _, s in buffers], np.int32) for i in (2, 3))
        state["strides"] = np.array([8, 16, 32, 64], np.int32)
        state["rows"] = np.zeros((n, MAX_DETECTIONS, 6), np.float32)
        state["counts"] = np.zeros(n, np.int32)
        state["slot"] = np.arange(MAX_DETECTIONS)[None, :]
    return state


# ---- what is called from outside --------------------------------------------------------------------------------------------

def prepare(case, seed):
    return _prepare_layer(case, seed) if case["kind"] == "layer" else _prepare_net(case, seed)


def run(state):
    s = state
    if s["kind"] == "layer":
        s["layer"].forward(s["x"].data_ptr(), s["src"], s["n"], s["h"], s["w"], s["y"].data_ptr(), s["dst"])
        return s["y"]
    if s["kind"] == "backbone":
        if s["mode"] == "host":
            return s["net"].forward("data", s["x"], ["conv5"])
        if s["mode"] == "pinned":
            s["net"].forward_raw("data", C.c_void_p(s["x"].data_ptr()), False, s["shape"], ["conv5"], [s["y"].data_ptr()])
            return s["y"]
        s["graph"].launch()
        return s["outputs"]
    if s["mode"] == "host":
        rows, count = s["net"].forward_rows("data", s["x"], "nanodet")
        table = np.zeros((s["cells"], 6), np.float32)  # one shape whatever the image shows
        table[:count] = rows
        return {"rows": table, "count": count}
    s["graph"].launch()
    ctx, rows, counts = s["ctx"], s["rows"], s["counts"]
    ctx.check(ctx.lib.ott_nanodet_detect(ctx.h, s["heads"], s["grid_h"].ctypes.data, s["grid_w"].ctypes.data, s["strides"].ctypes.data, len(s["strides"]),
                                         s["shape"][0], CLASSES, REG_BINS, PROB_THRESHOLD, NMS_THRESHOLD, rows.ctypes.data, counts.ctypes.data,
                                         MAX_DETECTIONS))
    rows[s["slot"] >= counts[:, None]] = 0.0  # rows past an image's count mean nothing
    return {"heads": s["outputs"], "rows": rows, "counts": counts}


def work(case):
    n, h, w = case["n"], case["h"], case["w"]
    if case["kind"] == "layer":
        oh, ow = _out_hw(case)
        taps = (1 if case["depthwise"] else case["cin"]) * case["k"] ** 2
        return dict(bytes=n * case["cin"] * h * w * (4 if case["src"] == "f32" else 1) + n * case["cout"] * oh * ow * (4 if case["dst"] == "f32" else 1) +
                    case["cout"] * taps, flops=2 * n * case["cout"] * taps * oh * ow)
    layers = _layers(case, h, w)
    sizes, macs = graphs.conv_input_hw(layers, h, w)
    geometry = graphs.conv_geometry(layers)
    weights = sum(g["cout"] * (g["cin"] // g["groups"]) * g["k"] ** 2 for g in geometry.values())
    ends = ["conv5"] if case["kind"] == "backbone" else list(graphs.NANODET_OUTPUTS)
    results = sum(geometry[e]["cout"] * math.prod(sizes[e]) for e in ends) if case["kind"] == "backbone" or case["mode"] == "graph" else 0  # 1x1 layers
    return dict(bytes=4 * n * (3 * h * w + results) + weights, flops=2 * n * macs)


def tolerance(case):
    # Everything in front of the decode is exact: s32 sums and a fixed order of fp32 roundings behind them. The decode's exp and
    # divisions may round differently in the last place, which moves a box coordinate of a few hundred pixels by about 1e-5.
    return {"rel": 1e-5, "max": 1e-4} if case["kind"] == "detector" else "exact"
