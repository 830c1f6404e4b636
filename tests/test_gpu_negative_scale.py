"""GPU: requantizing layers with output scales of both signs behind ReLU and ReLU6 (what is rounded is then below zero), both rounding
rules, bit for bit against the CPU checker: the dense kernel's one-tile and specialised builds, the depthwise kernels and the fused pair
and unit; and a scale that is infinite."""
import ctypes as C

import numpy as np
import pytest

from support import ACT_NONE, ACT_RELU, ACT_RELU6, ROUND_ADD_HALF_TRUNC, ROUND_HALF_AWAY, ConvCase, nchw_to_nhwc_padded, nhwc_padded_to_nchw, run_port

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from tensor_b200 import Context
    with Context(0) as c:
        yield c


@pytest.mark.parametrize("rounding", [ROUND_ADD_HALF_TRUNC, ROUND_HALF_AWAY])
@pytest.mark.parametrize("act", [ACT_RELU, ACT_RELU6])
@pytest.mark.parametrize("cin,k,stride,n,h,depthwise", [(40, 1, 1, 1, 9, False), (40, 1, 1, 90, 20, False), (40, 3, 1, 2, 20, False), (48, 3, 1, 2, 17, True),
                                                         (48, 3, 2, 2, 17, True), (33, 5, 1, 2, 14, True)])
def test_scales_of_both_signs(ctx, rounding, act, cin, k, stride, n, h, depthwise):
    from gpu_support import bits, run_gpu
    case = ConvCase(f"neg_{cin}_{k}", cin, cin, k, stride, k // 2, groups=cin if depthwise else 1, n=n, h=h, w=h, int8_scale_term=101, act_type=act,
                    s8_input=True, w_std=0.5 if depthwise else 0.1, seed=cin + k).make()
    scale = np.geomspace(0.5, 300.0, cin).astype(np.float32)
    case.out_scales = np.where(np.arange(cin) % 3 == 0, scale, -scale).astype(np.float32)
    got, want = run_gpu(ctx, case, rounding, want_acc=False)["y"], run_port(case, rounding, want_acc=False)["y"]
    assert want.min() == -127 and want.max() == 127 and np.unique(want).size > 100
    assert np.array_equal(bits(got), bits(want))


@pytest.mark.parametrize("act", [ACT_RELU, ACT_RELU6])
@pytest.mark.parametrize("unit,f32_out", [(False, False), (True, False), (True, True)])
def test_fused_layers(ctx, act, unit, f32_out):
    """1x1 layers with scales of both signs before and behind a depthwise layer, in the fused kernels."""
    from gpu_support import bits, make_layer
    from tensor_b200 import F32_NCHW, S8_NHWC, DwPwInt8, UnitInt8, nhwc_channels
    c, n, h, w = 40, 2, 17, 20
    signs = np.where(np.arange(c) % 3 == 0, 1, -1) * np.geomspace(2.0, 1200.0, c)
    common = dict(n=n, h=h, w=w, bias_term=1, s8_input=True)
    pw1 = ConvCase("neg_pw1", c, c, 1, 1, 0, int8_scale_term=101, act_type=act, w_std=0.1, seed=1, **common).make()
    dw = ConvCase("neg_dw", c, c, 3, 1, 1, groups=c, int8_scale_term=101, act_type=ACT_NONE, w_std=0.5, seed=2, **common).make()
    pw2 = ConvCase("neg_pw2", c, c, 1, 1, 0, int8_scale_term=1 if f32_out else 101, act_type=act, w_std=0.1, seed=3, **common).make()
    pw1.out_scales = signs.astype(np.float32)
    if not f32_out:
        pw2.out_scales = signs[::-1].astype(np.float32)
    if unit:
        dw.x_s8 = run_port(pw1, ROUND_ADD_HALF_TRUNC, want_acc=False)["y"]
        assert dw.x_s8.min() == -127 and dw.x_s8.max() == 127
    pw2.x_s8 = run_port(dw, ROUND_ADD_HALF_TRUNC, want_acc=False)["y"]
    want = run_port(pw2, ROUND_ADD_HALF_TRUNC, want_acc=False)["y"]
    assert f32_out or (want.min() == -127 and want.max() == 127 and np.unique(want).size > 100)
    layers = [make_layer(ctx, x, ROUND_ADD_HALF_TRUNC) for x in ((pw1, dw, pw2) if unit else (dw, pw2))]
    fused = (UnitInt8 if unit else DwPwInt8)(ctx, *layers)
    dtype = F32_NCHW if f32_out else S8_NHWC
    out = layers[-1].out_array(n, h, w, dtype)
    x, y = ctx.to_device(nchw_to_nhwc_padded((pw1 if unit else dw).x_s8, nhwc_channels(c))), ctx.malloc(out.nbytes)
    fused.forward_io(n, h, w, y, dtype, in_dev=x)
    got = ctx.to_host(y, out.shape, out.dtype)
    assert np.array_equal(bits(got if f32_out else nhwc_padded_to_nchw(got, c)), bits(want))
    for p in (x, y):
        ctx.free(p)
    for o in (fused, *layers):
        o.close()


@pytest.mark.parametrize("negative", [False, True])
def test_fused_pair_refuses_a_negative_depthwise_scale(ctx, negative):
    from gpu_support import make_layer
    from tensor_b200 import DwPwInt8, OtterB200Error
    dw = ConvCase("refused_dw", 40, 40, 3, 1, 1, groups=40, bias_term=1, int8_scale_term=101, act_type=ACT_NONE, s8_input=True, n=1, h=8, w=8, seed=2).make()
    pw = ConvCase("refused_pw", 40, 40, 1, 1, 0, bias_term=1, int8_scale_term=101, act_type=ACT_RELU, s8_input=True, n=1, h=8, w=8, seed=3).make()
    dw.out_scales = np.linspace(1.0, 40.0, 40).astype(np.float32)
    if negative:
        dw.out_scales[7] = -3.0
    layers = [make_layer(ctx, x, ROUND_ADD_HALF_TRUNC) for x in (dw, pw)]
    if negative:
        with pytest.raises(OtterB200Error):
            DwPwInt8(ctx, *layers)
    else:
        DwPwInt8(ctx, *layers).close()
    for layer in layers:
        layer.close()


def test_first_layer_maxpool_with_negative_scales(ctx):
    """Against the fp32 form of the same kernel, rounded half away from zero."""
    from tensor_b200 import ConvInt8, nhwc_channels
    n, h, w, cout = 1, 32, 40, 24
    case = ConvCase("stem", 3, cout, 3, stride=2, pad=1, n=n, h=h, w=w, int8_scale_term=2, act_type=ACT_RELU, x_lo=0.0, seed=3).make()
    scales = np.linspace(-60.0, 60.0, cout).astype(np.float32)
    kw = dict(cin=3, cout=cout, kh=3, kw=3, sh=2, sw=2, ph=1, pw=1, bias_term=1, act_type=ACT_RELU, rounding=ROUND_HALF_AWAY, weight=case.weight,
              bias=case.bias, w_scales=case.w_scales, in_scales=case.in_scales)
    f32_layer, s8_layer = ConvInt8(ctx, int8_scale_term=2, **kw), ConvInt8(ctx, int8_scale_term=101, out_scales=scales, **kw)
    oh, ow = f32_layer.out_hw(h, w)
    ph, pw, cp = (oh - 1) // 2 + 1, (ow - 1) // 2 + 1, nhwc_channels(cout)
    x, f, q = ctx.to_device(case.x_f32), ctx.malloc(n * cout * ph * pw * 4), ctx.malloc(n * ph * pw * cp)
    ctx.check(ctx.lib.ott_conv_int8_forward_maxpool(ctx.h, f32_layer.h, C.c_void_p(x), n, h, w, 0, C.c_void_p(f)))
    ctx.check(ctx.lib.ott_conv_int8_forward_maxpool_s8(ctx.h, s8_layer.h, C.c_void_p(x), n, h, w, 0, C.c_void_p(q)))
    t = ctx.to_host(f, (n, cout, ph, pw), np.float32) * scales[None, :, None, None]  # fp32 products, as in the kernel
    want = np.clip(np.trunc(t.astype(np.float64) + np.copysign(0.5, t)), -127, 127).astype(np.int8)
    assert want.min() < -5 and want.max() > 5
    assert np.array_equal(nhwc_padded_to_nchw(ctx.to_host(q, (n, ph, pw, cp), np.int8), cout), want)
    for p in (x, f, q):
        ctx.free(p)
    f32_layer.close()
    s8_layer.close()


def test_infinite_scale_leaves_the_padding_channels_zero(ctx):
    """A launch large enough for the build that takes one scale as a scalar; every real output saturates."""
    from tensor_b200 import S8_NHWC, ConvInt8
    rng, cin, cout, h, w = np.random.default_rng(4), 32, 20, 1024, 1024
    weight = rng.integers(-127, 128, size=(cout, cin, 1, 1), dtype=np.int8)
    layer = ConvInt8(ctx, cin=cin, cout=cout, kh=1, kw=1, int8_scale_term=101, weight=weight, bias=np.full(cout, 0.123, np.float32),
                     w_scales=np.full(cout, 50, np.float32), in_scales=np.full(1, 127, np.float32), out_scales=np.full(1, np.inf, np.float32))
    x, y = ctx.to_device(rng.integers(-127, 128, size=(1, h, w, cin), dtype=np.int8)), ctx.malloc(h * w * 32)
    layer.forward(x, S8_NHWC, 1, h, w, y, S8_NHWC)
    got = ctx.to_host(y, (h, w, 32), np.int8)
    assert not got[..., cout:].any() and (np.abs(got[..., :cout].astype(np.int32)) == 127).all()
    for p in (x, y):
        ctx.free(p)
    layer.close()
