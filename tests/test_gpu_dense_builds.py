"""GPU: fp32 input quantized inside the dense tensor-core kernel with several tiles per CTA (the stage ring wraps, the last tile is
ragged), bit for bit against the CPU checker."""
import numpy as np
import pytest

from support import ACT_LRELU, ACT_NONE, ACT_RELU, ACT_RELU6, ROUND_ADD_HALF_TRUNC, ConvCase, nhwc_padded_to_nchw, run_port

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
