"""GPU: requantizing layers with output scales of both signs behind ReLU and ReLU6 (what is rounded is then below zero), both rounding
rules, bit for bit against the CPU checker: the dense kernel's one-tile and specialised builds and the depthwise kernels; and a scale
that is infinite."""
import ctypes as C

import numpy as np
import pytest

from support import ACT_RELU, ACT_RELU6, ROUND_ADD_HALF_TRUNC, ROUND_HALF_AWAY, ConvCase, nhwc_padded_to_nchw, run_port

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
