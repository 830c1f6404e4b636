"""GPU: the 3-channel first layer, alone and with its max-pool, on an image that starts on every 4-byte offset from a 16-byte boundary:
the bytes of the aligned run, both rounding rules; and batches whose CTAs each walk over several tiles, the image by boxes and pixel
by pixel; and a LeakyReLU whose slope is negative, which no maximum of sums goes through."""
import ctypes as C

import numpy as np
import pytest

from support import ACT_LRELU, ACT_RELU, ROUND_ADD_HALF_TRUNC, ROUND_HALF_AWAY, ConvCase, run_port

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from tensor_b200 import Context
    with Context(0) as c:
        yield c


@pytest.mark.parametrize("stride", [1, 2])
@pytest.mark.parametrize("rounding", [ROUND_ADD_HALF_TRUNC, ROUND_HALF_AWAY])
@pytest.mark.parametrize("offset", [1, 2, 3])
def test_first_layer_on_a_misaligned_image(ctx, stride, rounding, offset):
    from gpu_support import bits, make_layer
    from tensor_b200 import F32_NCHW
    n, h, w, cout = 2, 12, 20, 24
    case = ConvCase("stem_offset", 3, cout, 3, stride, 1, n=n, h=h, w=w, int8_scale_term=2, act_type=ACT_RELU, x_lo=0.0, seed=3).make()
    want = run_port(case, rounding, want_acc=False)["y"]
    layer = make_layer(ctx, case, rounding)
    padded = np.zeros(case.x_f32.size + 4, np.float32)
    padded[offset:offset + case.x_f32.size] = case.x_f32.reshape(-1)
    x, aligned, y = ctx.to_device(padded), ctx.to_device(case.x_f32), ctx.malloc(want.nbytes)
    layer.forward(x + 4 * offset, F32_NCHW, n, h, w, y, F32_NCHW)
    assert np.array_equal(bits(ctx.to_host(y, want.shape, np.float32)), bits(want))
    oh, ow = (want.shape[2] - 1) // 2 + 1, (want.shape[3] - 1) // 2 + 1
    pooled = []
    for p in (aligned, x + 4 * offset):
        ctx.check(ctx.lib.ott_conv_int8_forward_maxpool(ctx.h, layer.h, C.c_void_p(p), n, h, w, 0, C.c_void_p(y)))
        pooled.append(ctx.to_host(y, (n, cout, oh, ow), np.float32))
    assert np.array_equal(bits(pooled[0]), bits(pooled[1]))
    for p in (x, aligned, y):
        ctx.free(p)
    layer.close()


@pytest.mark.parametrize("stride", [1, 2])
@pytest.mark.parametrize("w,offset", [(72, 0), (70, 0), (71, 0), (72, 1)])
def test_first_layer_and_maxpool_over_several_tiles(ctx, stride, w, offset):
    """More than twice the tiles that the GPU's CTAs hold at once; the first, the middle and the last image against the checker."""
    from gpu_support import bits
    from graph_walk import maxpool_nchw
    from support import nhwc_padded_to_nchw
    from tensor_b200 import ConvInt8, nhwc_channels
    n, h, cout = 91 if stride == 1 else 233, 50, 24
    case = ConvCase("stem_tiles", 3, cout, 3, stride, 1, n=3, h=h, w=w, int8_scale_term=2, act_type=ACT_RELU, x_lo=0.0, seed=5).make()
    conv = run_port(case, ROUND_ADD_HALF_TRUNC, want_acc=False)["y"]
    want = maxpool_nchw(conv, 3, 2, 1, pad_zero=False)
    scales = np.linspace(20.0, 60.0, cout).astype(np.float32)
    t = want * scales[None, :, None, None]  # fp32 products, as in the kernel
    want_s8 = np.clip(np.trunc(t.astype(np.float64) + 0.5), -127, 127).astype(np.int8)
    oh, ow = want.shape[2:]
    assert n * ((oh + 5) // 6) * ((ow + 15) // 16) > 2 * 4 * 148
    x = np.tile(np.random.default_rng(6).uniform(0, 1, size=(5, 3, h, w)).astype(np.float32), (n // 5 + 1, 1, 1, 1))[:n]
    at = [0, n // 2, n - 1]
    x[at] = case.x_f32
    kw = dict(cin=3, cout=cout, kh=3, kw=3, sh=stride, sw=stride, ph=1, pw=1, bias_term=1, act_type=ACT_RELU, weight=case.weight, bias=case.bias,
              w_scales=case.w_scales, in_scales=case.in_scales)
    f32_layer, s8_layer = ConvInt8(ctx, int8_scale_term=2, **kw), ConvInt8(ctx, int8_scale_term=101, out_scales=scales, **kw)
    image = ctx.to_device(np.concatenate([np.zeros(offset, np.float32), x.reshape(-1)]))
    f, q = ctx.malloc(n * cout * oh * ow * 4), ctx.malloc(n * oh * ow * nhwc_channels(cout))
    ctx.check(ctx.lib.ott_conv_int8_forward_maxpool(ctx.h, f32_layer.h, C.c_void_p(image + 4 * offset), n, h, w, 0, C.c_void_p(f)))
    ctx.check(ctx.lib.ott_conv_int8_forward_maxpool_s8(ctx.h, s8_layer.h, C.c_void_p(image + 4 * offset), n, h, w, 0, C.c_void_p(q)))
    got, got_s8 = ctx.to_host(f, (n, cout, oh, ow), np.float32), ctx.to_host(q, (n, oh, ow, nhwc_channels(cout)), np.int8)
    assert np.array_equal(bits(got[at]), bits(want)) and np.array_equal(nhwc_padded_to_nchw(got_s8[at], cout), want_s8)
    rest = [i for i in range(n - 5) if i not in at and i + 5 not in at]  # images repeat every five
    assert all(np.array_equal(got[i], got[i + 5]) and np.array_equal(got_s8[i], got_s8[i + 5]) for i in rest)
    for p in (image, f, q):
        ctx.free(p)
    f32_layer.close()
    s8_layer.close()


@pytest.mark.parametrize("pad_zero", [0, 1])
def test_maxpool_behind_a_negative_slope(ctx, pad_zero):
    from gpu_support import bits
    from graph_walk import maxpool_nchw
    from support import nhwc_padded_to_nchw
    from tensor_b200 import ConvInt8, nhwc_channels
    n, h, w, cout = 2, 30, 44, 20
    case = ConvCase("stem_slope", 3, cout, 3, 2, 1, n=n, h=h, w=w, int8_scale_term=2, act_type=ACT_LRELU, act_param0=-0.5, seed=7).make()
    want = maxpool_nchw(run_port(case, ROUND_ADD_HALF_TRUNC, want_acc=False)["y"], 3, 2, 1, pad_zero=bool(pad_zero))
    scales = np.linspace(20.0, 60.0, cout).astype(np.float32)
    t = want * scales[None, :, None, None]
    want_s8 = np.clip(np.trunc(t.astype(np.float64) + np.copysign(0.5, t)), -127, 127).astype(np.int8)
    kw = dict(cin=3, cout=cout, kh=3, kw=3, sh=2, sw=2, ph=1, pw=1, bias_term=1, act_type=ACT_LRELU, act_param0=-0.5, weight=case.weight, bias=case.bias,
              w_scales=case.w_scales, in_scales=case.in_scales)
    f32_layer, s8_layer = ConvInt8(ctx, int8_scale_term=2, **kw), ConvInt8(ctx, int8_scale_term=101, out_scales=scales, **kw)
    oh, ow = want.shape[2:]
    x, f, q = ctx.to_device(case.x_f32), ctx.malloc(n * cout * oh * ow * 4), ctx.malloc(n * oh * ow * nhwc_channels(cout))
    ctx.check(ctx.lib.ott_conv_int8_forward_maxpool(ctx.h, f32_layer.h, C.c_void_p(x), n, h, w, pad_zero, C.c_void_p(f)))
    ctx.check(ctx.lib.ott_conv_int8_forward_maxpool_s8(ctx.h, s8_layer.h, C.c_void_p(x), n, h, w, pad_zero, C.c_void_p(q)))
    assert np.array_equal(bits(ctx.to_host(f, want.shape, np.float32)), bits(want))
    assert np.array_equal(nhwc_padded_to_nchw(ctx.to_host(q, (n, oh, ow, nhwc_channels(cout)), np.int8), cout), want_s8)
    for p in (x, f, q):
        ctx.free(p)
    f32_layer.close()
    s8_layer.close()
