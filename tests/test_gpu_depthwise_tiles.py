"""GPU: the CUDA-core depthwise kernel at the edges of its tiles, bit for bit against the CPU checker: widths around its 4-column
groups, its column tiles and its bands; fp32 rows that start on every offset from a 16-byte boundary; channel counts around its
groups; both filter sizes, strides and roundings; fp32 and int8 on either side; a channel range of a wider tensor; and layers
gathered in 32-channel groups on launches too small for the tensor cores."""
import ctypes as C

import numpy as np
import pytest

from support import ACT_LRELU, ACT_NONE, ACT_RELU, ROUND_ADD_HALF_TRUNC, ROUND_HALF_AWAY, ConvCase, run_port

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from tensor_b200 import Context
    with Context(0) as c:
        yield c


@pytest.mark.parametrize("s8_input", [False, True], ids=["f32", "s8"])
@pytest.mark.parametrize("k,stride", [(3, 1), (3, 2), (5, 1), (5, 2)])
@pytest.mark.parametrize("c,n,h,w", [(2, 1, 1, 1), (3, 2, 2, 3), (33, 1, 5, 7), (16, 3, 13, 13), (40, 2, 9, 66), (20, 1, 70, 5), (31, 2, 26, 81),
                                     (64, 1, 34, 65), (48, 5, 41, 44)])
def test_tile_edges(ctx, c, n, h, w, k, stride, s8_input):
    from gpu_support import bits, run_gpu
    for term, act, rounding in ((101, ACT_RELU, ROUND_ADD_HALF_TRUNC), (101, ACT_LRELU, ROUND_HALF_AWAY), (1, ACT_NONE, ROUND_ADD_HALF_TRUNC)):
        case = ConvCase(f"dwt_{c}_{h}_{w}", c, c, k, stride, k // 2, groups=c, n=n, h=h, w=w, int8_scale_term=term, act_type=act,
                        act_param0=0.1, w_std=0.1, s8_input=s8_input, seed=c + h + w).make()
        ctx.check(ctx.lib.ott_set_depthwise_tensor_cores(ctx.h, 0))
        got = run_gpu(ctx, case, rounding, want_acc=False)["y"]
        ctx.check(ctx.lib.ott_set_depthwise_tensor_cores(ctx.h, 1))
        assert np.array_equal(bits(got), bits(run_port(case, rounding, want_acc=False)["y"]))


@pytest.mark.parametrize("k,c,n,h,w", [(3, 40, 31, 41, 45), (5, 40, 31, 41, 45), (5, 33, 100, 66, 10), (3, 64, 110, 60, 64)])
def test_large_fp32_outputs(ctx, k, c, n, h, w):
    """8 MB of rows that are not 16-byte aligned and 100 MB of aligned ones: the low bands, with and without row groups; four images each."""
    from gpu_support import bits, make_layer
    from support import nchw_to_nhwc_padded
    from tensor_b200 import F32_NCHW, S8_NHWC, nhwc_channels
    case = ConvCase(f"dwt_low_{k}_{w}", c, c, k, 1, k // 2, groups=c, n=n, h=h, w=w, int8_scale_term=1, act_type=ACT_RELU, w_std=0.1, s8_input=True, seed=c + w).make()
    layer = make_layer(ctx, case, ROUND_ADD_HALF_TRUNC)
    ctx.check(ctx.lib.ott_set_depthwise_tensor_cores(ctx.h, 0))
    got = layer.forward_host(nchw_to_nhwc_padded(case.x_s8, nhwc_channels(c)), S8_NHWC, F32_NCHW)
    ctx.check(ctx.lib.ott_set_depthwise_tensor_cores(ctx.h, 1))
    layer.close()
    some = [0, 1, n // 2, n - 1]
    case.n, case.x_s8 = len(some), np.ascontiguousarray(case.x_s8[some])
    assert np.array_equal(bits(got[some]), bits(run_port(case, ROUND_ADD_HALF_TRUNC, want_acc=False)["y"]))


@pytest.mark.parametrize("first,total", [(1, 7), (2, 6), (3, 6)])
def test_channel_range_on_every_alignment(ctx, first, total):
    """Planes of an odd size inside a wider tensor: every plane starts at another offset from a 16-byte boundary."""
    from gpu_support import bits, make_layer
    from tensor_b200 import F32_NCHW
    c, n, h, w = 3, 2, 7, 9
    case = ConvCase("dwt_range", c, c, 3, 1, 1, groups=c, n=n, h=h, w=w, int8_scale_term=1, w_std=0.1, seed=9).make()
    wide = np.random.default_rng(1).uniform(-1, 1, size=(n, total, h, w)).astype(np.float32)
    case.x_f32 = np.ascontiguousarray(wide[:, first:first + c])
    want = run_port(case, 0, want_acc=False)["y"]
    layer = make_layer(ctx, case, 0)
    x, y = ctx.to_device(wide), ctx.malloc(want.nbytes)
    ctx.check(ctx.lib.ott_conv_int8_forward_ex(ctx.h, layer.h, C.c_void_p(x + 4 * first * h * w), F32_NCHW, total, n, h, w, C.c_void_p(y), F32_NCHW, None))
    got = ctx.to_host(y, want.shape, np.float32)
    ctx.free(x)
    ctx.free(y)
    layer.close()
    assert np.array_equal(bits(got), bits(want))


@pytest.mark.parametrize("stride,h,w", [(1, 6, 5), (2, 11, 9)])
def test_gathered_in_wide_groups_on_a_small_map(ctx, stride, h, w):
    """Sources of 48 and 58 channels: the last 32-channel group of the first one reaches past its channel stride."""
    from tensor_b200 import S8_NHWC, ConvInt8, nhwc_channels
    rng = np.random.default_rng(stride)
    source_channels, n = [48, 58], 2
    pick = [(0, i) for i in range(33, 48)] + [(1, i) for i in range(0, 58, 2)]
    c = len(pick)
    case = ConvCase("dwt_gather", c, c, 3, stride, 1, groups=c, n=n, h=h, w=w, int8_scale_term=101, act_type=ACT_NONE, w_std=0.1, s8_input=True, seed=5).make()
    case.in_scales = np.full_like(case.in_scales, case.in_scales[0])
    srcs = [rng.integers(-127, 128, size=(n, h, w, nhwc_channels(sc)), dtype=np.int8) for sc in source_channels]
    case.x_s8 = np.ascontiguousarray(np.stack([srcs[s][..., i] for s, i in pick], axis=1))
    want = run_port(case, 0, want_acc=False)["y"]
    layer = ConvInt8(ctx, cin=c, cout=c, kh=3, kw=3, sh=stride, sw=stride, ph=1, pw=1, groups=c, int8_scale_term=101, weight=case.weight, bias=case.bias,
                     w_scales=case.w_scales, in_scales=case.in_scales[:1], out_scales=case.out_scales,
                     gathered=(source_channels, [s for s, _ in pick], [i for _, i in pick]))
    stored, pos = layer.gathered_layout()
    assert stored % 32 == 0
    dev = [ctx.to_device(a) for a in srcs]
    oh, ow = layer.out_hw(h, w)
    y = ctx.malloc(n * oh * ow * stored)
    layer.forward_io(n, h, w, y, S8_NHWC, sources=dev)
    got = ctx.to_host(y, (n, oh, ow, stored), np.int8)
    for p in dev + [y]:
        ctx.free(p)
    layer.close()
    assert np.array_equal(got[..., pos].transpose(0, 3, 1, 2), want)
    assert not np.delete(got, pos, axis=3).any()
