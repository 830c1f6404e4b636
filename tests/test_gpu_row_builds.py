"""GPU: int8 launches of the dense tensor-core kernel with output channels as accumulator rows, bit for bit against the CPU checker: one
and several accumulators per panel, 64-row ones, several panels, ragged last tiles, every epilogue, and a start long before the previous
kernel ends."""
import numpy as np
import pytest

from support import ACT_LRELU, ACT_NONE, ACT_RELU, ACT_RELU6, ROUND_ADD_HALF_TRUNC, ROUND_HALF_AWAY, ConvCase, run_port

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from tensor_b200 import Context
    with Context(0) as c:
        yield c


def _check(ctx, case, rounding=ROUND_ADD_HALF_TRUNC, scale=None):
    from gpu_support import bits, run_gpu
    case.make()
    if scale is not None:
        case.out_scales = scale
    got, want = run_gpu(ctx, case, rounding, want_acc=False), run_port(case, rounding, want_acc=False)
    assert np.array_equal(bits(got["y"]), bits(want["y"]))
    assert not got["y_pad"].any()


def _case(cin, cout, n, h, w, act):
    return ConvCase(f"rows_{cin}_{cout}", cin, cout, 1, 1, 0, n=n, h=h, w=w, bias_term=1, int8_scale_term=101, act_type=act, act_param0=0.1, s8_input=True,
                    w_std=0.5, seed=cin + cout)


@pytest.mark.parametrize("cin,cout,panels", [(58, 58, (64, 64)), (340, 64, (64, 64)), (64, 96, (128, 128)), (116, 116, (128, 128)), (96, 176, (192, 192)),
                                             (128, 192, (192, 192)), (232, 232, (128, 256)), (40, 352, (128, 192)), (200, 464, (128, 256)), (512, 480, (256, 256)),
                                             (130, 992, (256, 256))])
def test_pointwise(ctx, cin, cout, panels):
    for n, panel in zip((7, 41), panels):  # 177 and 1036 tiles, the last one ragged: about one and seven per CTA
        assert ctx.lib.ott_debug_dense_rows(cin, cout, n, 61, 53, 0, 148) == panel
        _check(ctx, _case(cin, cout, n, 61, 53, ACT_RELU))


@pytest.mark.parametrize("act", [ACT_NONE, ACT_RELU, ACT_LRELU, ACT_RELU6])
@pytest.mark.parametrize("scale", [0.2, 21.25, 3e6, -0.3])  # the third leaves 16 bits
def test_epilogues(ctx, act, scale):
    for rounding, per_channel in ((ROUND_ADD_HALF_TRUNC, False), (ROUND_HALF_AWAY, True)):
        cout = 180
        assert ctx.lib.ott_debug_dense_rows(64, cout, 7, 61, 53, 0, 148) == 192
        s = (scale * np.linspace(0.97, 1.03, cout)).astype(np.float32) if per_channel else np.full(1, scale, np.float32)
        _check(ctx, _case(64, cout, 7, 61, 53, act), rounding, s)


@pytest.mark.parametrize("cin,cout,h,w", [(256, 512, 44, 20), (40, 330, 44, 21), (130, 240, 20, 44), (33, 64, 44, 20), (64, 100, 46, 22), (100, 16, 44, 20), (17, 40, 44, 20), (24, 24, 12, 10),
                                          (32, 384, 20, 18)])
@pytest.mark.parametrize("act", [ACT_RELU6, ACT_NONE])
def test_quantized_inside(ctx, cin, cout, h, w, act):
    """fp32 input of 100 MB: one to four accumulators per tile of 64 pixels, the last tile of an image ragged; the first, the middle and
    the last image against the checker. From two boxes of 16 channels per tile on, so that most of the warps that quantize have none."""
    from gpu_support import make_layer
    from tensor_b200 import F32_NCHW, S8_NHWC, nhwc_channels
    from support import nhwc_padded_to_nchw
    n = (100 << 20) // (4 * cin * h * w) + 1
    assert ctx.lib.ott_debug_dense_rows(cin, cout, n, h, w, 1, 148) == (cout + 63) // 64 * 64
    case = _case(cin, cout, 3, h, w, act)
    case.s8_input = False
    case.make()
    x = np.tile(np.random.default_rng(cin).uniform(-1, 1, size=(7, cin, h, w)).astype(np.float32), (n // 7 + 1, 1, 1, 1))[:n]
    at = [0, n // 2, n - 1]
    x[at] = case.x_f32
    layer = make_layer(ctx, case, ROUND_ADD_HALF_TRUNC)
    dx, shape = ctx.to_device(x), (n, h, w, nhwc_channels(cout))
    y = ctx.malloc(int(np.prod(shape)))
    layer.forward(dx, F32_NCHW, n, h, w, y, S8_NHWC)
    got = ctx.to_host(y, shape, np.int8)
    assert np.array_equal(nhwc_padded_to_nchw(got[at], cout), run_port(case, ROUND_ADD_HALF_TRUNC, want_acc=False)["y"])
    assert np.array_equal(got[1:8], got[8:15]) and not got[..., cout:].any()
    layer.close()
    ctx.free(dx)
    ctx.free(y)


@pytest.mark.parametrize("f32", [False, True])
def test_waits_do_not_count_the_previous_kernel(ctx, f32):
    """A launch of several milliseconds that leaves SMs idle (eight panels: 144 of 148 CTAs), the next one's first CTAs beside it, and
    waits limited to one millisecond. The long launch's output is not looked at."""
    from gpu_support import make_layer
    from tensor_b200 import F32_NCHW, S8_NHWC, ConvInt8, nhwc_channels
    from support import nchw_to_nhwc_padded, nhwc_padded_to_nchw
    assert ctx.lib.ott_debug_dense_rows(512, 2048, 1, 1600, 1600, 0, 148) == 256
    rng = np.random.default_rng(2)
    before = ConvInt8(ctx, cin=512, cout=2048, kh=1, kw=1, int8_scale_term=101, act_type=ACT_RELU, weight=rng.integers(-127, 128, (2048, 512, 1, 1), dtype=np.int8),
                      bias=np.zeros(2048, np.float32), w_scales=np.full(2048, 50, np.float32), in_scales=np.full(1, 127, np.float32),
                      out_scales=np.full(1, 0.1, np.float32))
    n, h, w, cout = (320, 44, 20, 100) if f32 else (16, 52, 52, 100)
    cin = 96 if f32 else 64
    case = _case(cin, cout, 2, h, w, ACT_RELU)
    case.s8_input = not f32
    case.make()
    want = run_port(case, ROUND_ADD_HALF_TRUNC, want_acc=False)["y"]
    assert ctx.lib.ott_debug_dense_rows(cin, cout, n, h, w, int(f32), 148) == 128
    layer = make_layer(ctx, case, ROUND_ADD_HALF_TRUNC)
    one = case.x_f32 if f32 else nchw_to_nhwc_padded(case.x_s8, nhwc_channels(cin))
    x, shape = ctx.to_device(np.tile(one, (n // 2, 1, 1, 1))), (n, h, w, nhwc_channels(cout))
    y, big_x, big_y = ctx.malloc(int(np.prod(shape))), ctx.malloc(1600 * 1600 * 512), ctx.malloc(1600 * 1600 * 2048)
    ctx.memset(big_x, 1, 1600 * 1600 * 512)
    ctx.sync()
    ctx.check(ctx.lib.ott_set_wait_limit_ms(ctx.h, 1))
    for _ in range(3):
        before.forward(big_x, S8_NHWC, 1, 1600, 1600, big_y, S8_NHWC)
        layer.forward(x, F32_NCHW if f32 else S8_NHWC, n, h, w, y, S8_NHWC)
    ctx.sync()
    ctx.check(ctx.lib.ott_set_wait_limit_ms(ctx.h, 2000))
    got = ctx.to_host(y, shape, np.int8)
    for i in (0, n // 2, n - 2):
        assert np.array_equal(nhwc_padded_to_nchw(got[i:i + 2], cout), want)
    for p in (x, y, big_x, big_y):
        ctx.free(p)
    before.close()
    layer.close()
