"""GPU: the tensor-core convolution over narrow weight panels (launches with fewer pixel tiles than SMs), bit for bit against the
CPU checker: output widths around the panel widths, one tile and several, 1x1 and halo and strided filters, every output kind,
both roundings, with and without bias."""
import numpy as np
import pytest

from support import ACT_LRELU, ACT_NONE, ACT_RELU, ACT_RELU6, ROUND_ADD_HALF_TRUNC, ROUND_HALF_AWAY, ConvCase, run_port

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from tensor_b200 import Context
    with Context(0) as c:
        yield c


@pytest.mark.parametrize("k,stride", [(1, 1), (3, 1), (3, 2)])
@pytest.mark.parametrize("cin,cout,h,w", [(32, 17, 3, 5), (40, 33, 8, 16), (64, 64, 17, 9), (130, 65, 10, 10), (232, 240, 10, 10), (48, 129, 20, 21),
                                          (96, 300, 6, 7)])
def test_narrow_panels(ctx, cin, cout, h, w, k, stride):
    from gpu_support import bits, run_gpu
    for term, act, rounding, bias in ((101, ACT_RELU, ROUND_ADD_HALF_TRUNC, 1), (102, ACT_LRELU, ROUND_HALF_AWAY, 0), (101, ACT_NONE, ROUND_HALF_AWAY, 1),
                                      (1, ACT_RELU6, ROUND_ADD_HALF_TRUNC, 0)):
        case = ConvCase(f"panel_{cin}_{cout}", cin, cout, k, stride, k // 2, n=2, h=h, w=w, bias_term=bias, int8_scale_term=term, act_type=act,
                        act_param0=0.1, s8_input=True, seed=cin + cout + h).make()
        got, want = run_gpu(ctx, case, rounding), run_port(case, rounding)
        assert np.array_equal(got["acc"], want["acc"])
        assert np.array_equal(bits(got["y"]), bits(want["y"]))


@pytest.mark.parametrize("pixels", [(1, 1), (3, 5), (4, 4), (1, 17), (1, 31), (4, 8), (3, 11), (7, 9), (5, 13), (1, 127), (3, 43), (20, 20)])
@pytest.mark.parametrize("cin,cout", [(33, 40), (200, 70)])
def test_few_pixels_per_tile(ctx, cin, cout, pixels):
    from gpu_support import bits, run_gpu
    for term, s8_input, act in ((101, True, ACT_RELU), (1, True, ACT_RELU6), (101, False, ACT_LRELU), (1, False, ACT_NONE)):
        case = ConvCase(f"few_{pixels}", cin, cout, 1, 1, 0, n=1, h=pixels[0], w=pixels[1], bias_term=1, int8_scale_term=term, act_type=act, act_param0=0.1,
                        s8_input=s8_input, seed=cin + pixels[1]).make()
        got, want = run_gpu(ctx, case, ROUND_ADD_HALF_TRUNC), run_port(case, ROUND_ADD_HALF_TRUNC)
        assert np.array_equal(got["acc"], want["acc"])
        assert np.array_equal(bits(got["y"]), bits(want["y"]))


@pytest.mark.parametrize("k,pad", [(2, 0), (2, 1), (3, 0), (3, 1), (4, 1), (5, 2), (7, 3)])
@pytest.mark.parametrize("cin,cout,h,w,n", [(33, 20, 7, 9, 1), (64, 64, 31, 15, 3), (70, 40, 33, 17, 2), (130, 100, 35, 34, 1), (40, 48, 64, 65, 40)])
def test_stride_two_halo(ctx, cin, cout, h, w, n, k, pad):
    from gpu_support import bits, run_gpu
    for term, act in ((101, ACT_LRELU), (1, ACT_NONE)):
        case = ConvCase(f"s2_{k}_{cin}", cin, cout, k, 2, pad, n=n, h=h, w=w, bias_term=1, int8_scale_term=term, act_type=act, act_param0=0.1, s8_input=True,
                        seed=cin + k).make()
        got, want = run_gpu(ctx, case, ROUND_ADD_HALF_TRUNC), run_port(case, ROUND_ADD_HALF_TRUNC)
        assert np.array_equal(got["acc"], want["acc"])
        assert np.array_equal(bits(got["y"]), bits(want["y"]))
