"""GPU: requantized values on the edge between two integers. Every channel's output scale is chosen so that the product of one of its
values and the scale lies within a step or two of fp32 of n + 0.5, where one rounding of product and sum in place of two shows; bit for
bit against the CPU checker, in every kernel that requantizes, for every activation and both rules. And products next to 0.5 itself,
for which ReLU layers that round once are not taken."""
import numpy as np
import pytest

from support import (ACT_LRELU, ACT_NONE, ACT_RELU, ACT_RELU6, ROUND_ADD_HALF_TRUNC, ROUND_HALF_AWAY, ConvCase, nchw_to_nhwc_padded, nhwc_padded_to_nchw,
                     run_port)

pytestmark = pytest.mark.gpu
RULES = [ROUND_ADD_HALF_TRUNC, ROUND_HALF_AWAY]
ACTS = [ACT_NONE, ACT_RELU, ACT_LRELU, ACT_RELU6]


@pytest.fixture(scope="module")
def ctx():
    from tensor_b200 import Context
    with Context(0) as c:
        yield c


def _on_the_edge(case, rounding, low=1, high=126, seed=0):
    """Output scales for a case whose other parameters are made."""
    probe = case.int8_scale_term
    case.int8_scale_term = probe - 100
    v = run_port(case, rounding, want_acc=False)["y"]  # the activated values
    case.int8_scale_term = probe
    rng = np.random.default_rng(seed)
    scales = np.empty(case.cout, np.float32)
    for c in range(case.cout):
        seen = np.unique(v[:, c])
        seen = seen[(seen > 0.2 * seen.max()) & (seen > 0)]
        scales[c] = np.float32(rng.integers(low, high + 1) + 0.5) / (rng.choice(seen) if seen.size else np.float32(1.0))
    bits = scales.view(np.int32) + rng.integers(-2, 3, size=case.cout).astype(np.int32)
    case.out_scales = bits.view(np.float32)


def _make(name, cin, cout, k, act, n, h, w, s8_input, seed, stride=1, depthwise=False, std=0.05):
    # (small enough for ReLU6 not to cut most of them)
    return ConvCase(f"edge_{name}", cin, cout, k, stride, k // 2, groups=cin if depthwise else 1, n=n, h=h, w=w, bias_term=1, int8_scale_term=101, act_type=act,
                    act_param0=0.1, s8_input=s8_input, w_std=std, seed=seed).make()


@pytest.mark.parametrize("rounding", RULES)
@pytest.mark.parametrize("act", ACTS)
@pytest.mark.parametrize("name,cin,cout,k,stride,n,h,s8,depthwise", [
    ("one_tile", 64, 256, 1, 1, 1, 9, True, False), ("channel_rows", 64, 512, 1, 1, 16, 50, True, False), ("pixel_rows", 600, 256, 1, 1, 16, 50, True, False),
    ("inside", 96, 96, 1, 1, 10, 60, False, False), ("k3", 32, 128, 3, 1, 8, 50, True, False), ("k3_stride2", 64, 128, 3, 2, 16, 50, True, False),
    ("direct", 5, 7, 3, 1, 2, 9, True, False), ("dw3", 256, 256, 3, 1, 2, 20, True, True), ("dw3_f32", 256, 256, 3, 1, 2, 20, False, True),
    ("dw3_tensor", 256, 256, 3, 2, 20, 56, True, True), ("dw5", 256, 256, 5, 1, 2, 20, True, True), ("dw7", 64, 64, 7, 1, 2, 12, True, True)])
def test_layers(ctx, name, cin, cout, k, stride, n, h, s8, depthwise, act, rounding):
    from gpu_support import run_gpu
    for low, high in ((1, 126), (0, 0)):
        case = _make(name, cin, cout, k, act, n, h, h, s8, cin + k + act, stride, depthwise, 0.2 if depthwise else 0.05)
        _on_the_edge(case, rounding, low, high, seed=act)
        got, want = run_gpu(ctx, case, rounding, want_acc=False)["y"], run_port(case, rounding, want_acc=False)["y"]
        wrong = np.argwhere(got != want)
        assert not len(wrong), (low, len(wrong), [(tuple(i), int(got[tuple(i)]), int(want[tuple(i)])) for i in wrong[:5]])


@pytest.mark.parametrize("act", [ACT_RELU, ACT_RELU6])
@pytest.mark.parametrize("unit", [False, True])
def test_fused_layers(ctx, act, unit):
    from gpu_support import make_layer
    from tensor_b200 import S8_NHWC, DwPwInt8, UnitInt8, nhwc_channels
    for low, high in ((1, 126), (0, 0)):
        c, n, h, w = 64, 3, 17, 20
        pw1, dw, pw2 = _make("pw1", c, c, 1, act, n, h, w, True, 1), _make("dw", c, c, 3, ACT_NONE, n, h, w, True, 2, 1, True, 0.2), _make("pw2", c, c, 1, act, n, h, w, True, 3)
        if unit:
            _on_the_edge(pw1, ROUND_ADD_HALF_TRUNC, low, high, 1)
            dw.x_s8 = run_port(pw1, ROUND_ADD_HALF_TRUNC, want_acc=False)["y"]
        _on_the_edge(dw, ROUND_ADD_HALF_TRUNC, 100, 126, 2)
        pw2.x_s8 = run_port(dw, ROUND_ADD_HALF_TRUNC, want_acc=False)["y"]
        _on_the_edge(pw2, ROUND_ADD_HALF_TRUNC, low, high, 3)
        want = run_port(pw2, ROUND_ADD_HALF_TRUNC, want_acc=False)["y"]
        layers = [make_layer(ctx, x, ROUND_ADD_HALF_TRUNC) for x in ((pw1, dw, pw2) if unit else (dw, pw2))]
        fused = (UnitInt8 if unit else DwPwInt8)(ctx, *layers)
        out = layers[-1].out_array(n, h, w, S8_NHWC)
        x, y = ctx.to_device(nchw_to_nhwc_padded((pw1 if unit else dw).x_s8, nhwc_channels(c))), ctx.malloc(out.nbytes)
        fused.forward_io(n, h, w, y, S8_NHWC, in_dev=x)
        got = nhwc_padded_to_nchw(ctx.to_host(y, out.shape, out.dtype), c)
        assert np.array_equal(got, want), (low, np.argwhere(got != want)[:5])
        for p in (x, y):
            ctx.free(p)
        for o in (fused, *layers):
            o.close()


@pytest.mark.parametrize("rounding", RULES)
@pytest.mark.parametrize("k", [1, 3])
def test_quantized_input(ctx, rounding, k):
    """fp32 values next to n + 0.5 over the input scale, through a layer that hands them on (1x1 or depthwise, weight 1)."""
    from gpu_support import run_gpu
    c, n, h = 32, 4, 24
    rng = np.random.default_rng(k)
    case = _make("quantize", c, c, k, ACT_NONE, n, h, h, False, 5, 1, k == 3)
    case.weight[:] = 0
    for i in range(c):
        case.weight[i, 0 if k == 3 else i, k // 2, k // 2] = 1
    case.in_scales = np.full(c if k == 3 else 1, 37.3, np.float32)
    case.w_scales[:], case.bias[:] = 1.0, 0.0
    case.out_scales = np.full(c if k == 3 else 1, 37.3, np.float32)
    edge = ((rng.integers(-127, 127, size=case.x_f32.shape) + 0.5) / 37.3).astype(np.float32)
    case.x_f32 = (edge.view(np.int32) + rng.integers(-2, 3, size=edge.shape).astype(np.int32)).view(np.float32)
    got, want = run_gpu(ctx, case, rounding, want_acc=False)["y"], run_port(case, rounding, want_acc=False)["y"]
    assert np.array_equal(got, want) and np.unique(want).size > 200


@pytest.mark.parametrize("act", [ACT_RELU, ACT_RELU6])
@pytest.mark.parametrize("signs", [False, True])
@pytest.mark.parametrize("name,c,k,stride,n,h,s8,depthwise", [("dw3", 48, 3, 1, 2, 17, True, True), ("dw3_f32", 48, 3, 1, 2, 17, False, True),
                                                              ("dw3_tensor", 256, 3, 2, 20, 56, True, True), ("dw5", 48, 5, 2, 2, 17, True, True),
                                                              ("dw7", 48, 7, 1, 2, 12, True, True), ("one_tile", 64, 1, 1, 1, 9, True, False),
                                                              ("channel_rows", 64, 1, 1, 16, 50, True, False)])
def test_channels_switched_off(ctx, name, c, k, stride, n, h, s8, depthwise, signs, act):
    """A bias of -infinity leaves 0 of a channel behind ReLU and ReLU6, under scales of either sign."""
    from gpu_support import run_gpu
    case = _make(f"off_{name}", c, c, k, act, n, h, h, s8, c + k, stride, depthwise, 0.2 if depthwise else 0.05)
    case.bias[::5] = -np.inf
    scale = np.geomspace(5.0, 300.0, c).astype(np.float32)
    case.out_scales = np.where(np.arange(c) % 3 == 0, -scale, scale) if signs else scale
    got, want = run_gpu(ctx, case, ROUND_ADD_HALF_TRUNC, want_acc=False)["y"], run_port(case, ROUND_ADD_HALF_TRUNC, want_acc=False)["y"]
    assert not want[:, ::5].any() and np.unique(want).size > 50
    assert np.array_equal(got, want), np.argwhere(got != want)[:5]
