"""GPU: the requantizing epilogue on launches of one tile per CTA, bit for bit against the
CPU checker: activations that the int8 clamp carries out and ones
that it cannot (a ReLU6 whose 6 is not 127, sums that may leave 16 bits, a scale that saturates everything), one output scale and one
per channel, both roundings, with and without bias, sums of both signs."""
import numpy as np
import pytest

from support import ACT_LRELU, ACT_NONE, ACT_RELU, ACT_RELU6, ROUND_ADD_HALF_TRUNC, ROUND_HALF_AWAY, ConvCase, run_port

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from tensor_b200 import Context
    with Context(0) as c:
        yield c


@pytest.mark.parametrize("act", [ACT_NONE, ACT_RELU, ACT_LRELU, ACT_RELU6])
@pytest.mark.parametrize("scale", [0.2, 21.0, 21.25, 400.0, 3e6])  # six comes out as 1, 126, 127 and more; the last two leave 16 bits
@pytest.mark.parametrize("cin,cout,k,depthwise", [(64, 48, 1, False), (200, 300, 1, False), (33, 40, 3, False), (64, 64, 3, True), (40, 40, 5, True)])
def test_requantize_builds(ctx, act, scale, cin, cout, k, depthwise):
    from gpu_support import bits, run_gpu
    for rounding, per_channel, bias in ((ROUND_ADD_HALF_TRUNC, False, 1), (ROUND_HALF_AWAY, True, 0)):
        case = ConvCase(f"requant_{cin}_{cout}", cin, cout, k, 1, k // 2, groups=cin if depthwise else 1, n=2, h=11, w=13, bias_term=bias, int8_scale_term=101,
                        act_type=act, act_param0=0.1, s8_input=True, w_std=0.5, seed=cin + cout).make()
        case.out_scales = np.full(1, scale, np.float32)
        if per_channel:
            case.out_scales = (scale * np.linspace(0.97, 1.03, cout)).astype(np.float32)
        got, want = run_gpu(ctx, case, rounding), run_port(case, rounding)
        assert np.array_equal(bits(got["y"]), bits(want["y"]))
