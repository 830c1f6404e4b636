"""GPU: the 3-channel first layer, alone and with its max-pool, on an image that starts on every 4-byte offset from a 16-byte boundary:
the bytes of the aligned run, both rounding rules."""
import ctypes as C

import numpy as np
import pytest

from support import ACT_RELU, ROUND_ADD_HALF_TRUNC, ROUND_HALF_AWAY, ConvCase, run_port

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
