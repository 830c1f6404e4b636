"""GPU: builds of the dense tensor-core kernel that only larger launches take, bit for bit against the CPU checker: fp32 input quantized
inside with several tiles per CTA (the stage ring wraps, the last tile is ragged), the requantizing epilogues with several tiles per
CTA and panels wider than 32 columns, with pixels and with channels as accumulator rows, and the builds that take one output scale
as a scalar (sampled pixels)."""
import numpy as np
import pytest

from support import (ACT_LRELU, ACT_NONE, ACT_RELU, ACT_RELU6, ROUND_ADD_HALF_TRUNC, ROUND_HALF_AWAY, ConvCase, nchw_to_nhwc_padded, nhwc_padded_to_nchw,
                     run_port)

pytestmark = pytest.mark.gpu
SMS = 148


@pytest.fixture(scope="module")
def ctx():
    from tensor_b200 import Context
    with Context(0) as c:
        yield c


def _plan(lib, case):
    import ctypes as C
    out = (C.c_int * 8)()
    assert lib.ott_debug_dense_plan(case.cin, case.cout, case.k, case.stride, case.n, case.h, case.w, 0 if case.s8_input else 1, SMS, out) == 0
    return dict(zip(("tiles", "panels", "columns", "per_sm", "inside", "compact", "rows", "halo"), out))


@pytest.mark.parametrize("act", [ACT_NONE, ACT_RELU, ACT_LRELU, ACT_RELU6])
@pytest.mark.parametrize("cin,cout,term", [(116, 70, 101), (116, 70, 1), (200, 64, 101), (33, 150, 1)])
def test_quantized_inside_over_several_tiles(ctx, cin, cout, term, act):
    from gpu_support import bits, make_layer
    from tensor_b200 import F32_NCHW, S8_NHWC, nhwc_channels
    n, h, w = 13, 58, 62  # 46748 pixels: 365.2 tiles of 128, 3596 pixels an image
    case = ConvCase(f"inside_{cin}_{cout}", cin, cout, 1, 1, 0, n=n, h=h, w=w, bias_term=1, int8_scale_term=term, act_type=act, act_param0=0.1, seed=cin + act).make()
    p = _plan(ctx.lib, case)
    assert p["inside"] and p["tiles"] > 2 * SMS and p["panels"] == 1, p
    want = run_port(case, ROUND_ADD_HALF_TRUNC, want_acc=False)["y"]
    layer = make_layer(ctx, case, ROUND_ADD_HALF_TRUNC)
    flat = np.concatenate([np.zeros(1, np.float32), case.x_f32.reshape(-1)])
    for offset in (0, 1):  # wide loads, and an image that starts off a 16-byte boundary: pixel by pixel
        x = ctx.to_device(flat[1 - offset:])
        dtype = S8_NHWC if term > 100 else F32_NCHW
        shape = (n, h, w, nhwc_channels(cout)) if term > 100 else want.shape
        y = ctx.malloc(int(np.prod(shape)) * (1 if term > 100 else 4))
        layer.forward(x + 4 * offset, F32_NCHW, n, h, w, y, dtype)
        got = ctx.to_host(y, shape, np.int8 if term > 100 else np.float32)
        assert np.array_equal(bits(nhwc_padded_to_nchw(got, cout) if term > 100 else got), bits(want)), offset
        ctx.free(x)
        ctx.free(y)
    layer.close()


def _launch(lib, case):
    import ctypes as C
    out = (C.c_int * 9)()
    assert lib.ott_debug_dense_launch(case.cin, case.cout, case.k, case.stride, case.n, case.h, case.w, 0 if case.s8_input else 1, 1, SMS, out) == 0
    return dict(zip(("tiles", "panels", "columns", "per_sm", "inside", "compact", "rows", "halo", "channel_rows"), out))


def _differences(got, want):
    """How many outputs differ and where: a wrong 32 x 32 block points to an accumulator, a wrong piece of 512 KB to the host copies."""
    at = np.argwhere(got != want)
    first = [(tuple(int(v) for v in i), int(got[tuple(i)]), int(want[tuple(i)])) for i in at[:8]]
    return f"{len(at)} of {want.size} differ; images {sorted(set(at[:, 0]))[:8]}, channels {sorted(set(at[:, 1]))[:40]}; (image, channel, y, x), got, wanted: {first}"


@pytest.mark.parametrize("act", [ACT_NONE, ACT_RELU, ACT_LRELU, ACT_RELU6])
@pytest.mark.parametrize("scale", [0.2, 21.0, 21.25, 400.0, 3e6])  # six comes out as 1, 126, 127 and more; the last two leave 16 bits
@pytest.mark.parametrize("cin,cout,k,h,channel_rows", [(64, 96, 1, 52, 128), (40, 160, 1, 52, 128), (560, 96, 1, 52, 0), (33, 70, 3, 50, 0)])
def test_requantize_over_several_tiles(ctx, act, scale, cin, cout, k, h, channel_rows):
    from gpu_support import run_gpu
    for rounding, per_channel in ((ROUND_ADD_HALF_TRUNC, False), (ROUND_HALF_AWAY, True)):
        case = ConvCase(f"requant_{cin}_{cout}", cin, cout, k, 1, k // 2, n=16, h=h, w=h, bias_term=1, int8_scale_term=101, act_type=act, act_param0=0.1,
                        s8_input=True, w_std=0.5, seed=cin + cout).make()
        p = _launch(ctx.lib, case)
        assert not p["compact"] and p["columns"] > 32 and p["tiles"] > p["per_sm"] * SMS and p["channel_rows"] == channel_rows, p
        case.out_scales = np.full(1, scale, np.float32)
        if per_channel:
            case.out_scales = (scale * np.linspace(0.97, 1.03, cout)).astype(np.float32)
        got, want = run_gpu(ctx, case, rounding, want_acc=False)["y"], run_port(case, rounding, want_acc=False)["y"]
        assert np.array_equal(got, want), _differences(got, want)


@pytest.mark.parametrize("forward_host", [False, True])
def test_the_same_launch_many_times(ctx, forward_host):
    """64 -> 96 channels, 338 tiles, rounded half away from zero, 96 scales; with pixels as rows (an fp32 side output asks for that) and
    with channels as rows. Two hundred times from device buffers, or through the host copies."""
    from gpu_support import make_layer
    from tensor_b200 import F32_NCHW, S8_NHWC
    case = ConvCase("again", 64, 96, 1, 1, 0, n=16, h=52, w=52, bias_term=1, int8_scale_term=101, act_type=ACT_RELU, s8_input=True, w_std=0.5, seed=160).make()
    case.out_scales = (21.25 * np.linspace(0.97, 1.03, 96)).astype(np.float32)
    want = run_port(case, ROUND_HALF_AWAY, want_acc=False)["y"]
    layer = make_layer(ctx, case, ROUND_HALF_AWAY)
    x = nchw_to_nhwc_padded(case.x_s8, 64)
    if forward_host:
        for _ in range(200):
            got = nhwc_padded_to_nchw(layer.forward_host(x, S8_NHWC, S8_NHWC), 96)
            assert np.array_equal(got, want), _differences(got, want)
    else:
        shape, hw = (16, 52, 52, 96), 52 * 52
        xd, y, f = ctx.to_device(x), ctx.malloc(int(np.prod(shape))), ctx.malloc(16 * 96 * hw * 4)
        for i in range(200):
            ctx.memset(y, 0x55, int(np.prod(shape)))
            if i % 2:
                layer.forward(xd, S8_NHWC, 16, 52, 52, y, S8_NHWC)
            else:
                layer.forward_io(16, 52, 52, y, S8_NHWC, in_dev=xd, in_dtype=S8_NHWC, out_f32_dev=f, f32_channels=[3])
            got = nhwc_padded_to_nchw(ctx.to_host(y, shape, np.int8), 96)
            assert np.array_equal(got, want), _differences(got, want)
        for p in (xd, y, f):
            ctx.free(p)
    layer.close()


@pytest.mark.parametrize("act", [ACT_NONE, ACT_LRELU, ACT_RELU, ACT_RELU6])
@pytest.mark.parametrize("cin,cout,k", [(40, 64, 1), (560, 512, 1), (32, 64, 3), (64, 64, 3)])
def test_one_output_scale(ctx, act, cin, cout, k):
    """At least 2^25 outputs of one image; a band of rows in the middle and the last rows as images of their own for the checker."""
    from gpu_support import make_layer
    from tensor_b200 import S8_NHWC, nhwc_channels
    w = 520
    h = -(-(1 << 25) // (w * nhwc_channels(cout)))
    case = ConvCase(f"one_scale_{act}", cin, cout, k, 1, k // 2, n=1, h=h, w=w, bias_term=1, int8_scale_term=101, act_type=act, act_param0=0.1, s8_input=True,
                    w_std=0.5, seed=act + cin).make()
    assert h * w * nhwc_channels(cout) >= 1 << 25 and case.out_scales.size == 1
    p = _launch(ctx.lib, case)
    assert not p["compact"] and p["tiles"] > p["per_sm"] * SMS and (k == 1) == (p["halo"] == 0), p
    layer = make_layer(ctx, case, ROUND_ADD_HALF_TRUNC)
    got = nhwc_padded_to_nchw(layer.forward_host(nchw_to_nhwc_padded(case.x_s8, nhwc_channels(cin)), S8_NHWC, S8_NHWC), cout)
    layer.close()
    whole = case.x_s8
    for top in (h // 2, h - 12):
        case.h, case.x_s8 = 12, np.ascontiguousarray(whole[:, :, top:top + 12])
        want = run_port(case, ROUND_ADD_HALF_TRUNC, want_acc=False)["y"]
        a, b = (1, 11) if k == 3 else (0, 12)  # (the checker pads the band's own edges)
        assert np.array_equal(got[:, :, top + a:top + b], want[:, :, a:b]), _differences(got[:, :, top + a:top + b], want[:, :, a:b])
        assert np.unique(want).size > 50
