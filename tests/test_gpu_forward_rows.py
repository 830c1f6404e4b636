"""GPU: the detector's row-returning forward call after call: with changing images (from the third call of a shape on the heads come
from a replayed graph) against the CPU checker's decode, and with a bounded wait that ran out in front of the decode."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ERR_DEVICE_WAIT = -4


@pytest.fixture(scope="module")
def detector():
    from graph_support import build_net, oracle_conv, oracle_detect, wide_nanodet_case
    from graph_walk import walk
    from tensor_b200 import graphs
    L, params, x, _ = wide_nanodet_case()
    net = build_net(L + graphs.nanodet_plus_layers(64, 64, detect=True)[-1:], params)

    def want(image):
        from graph_support import oracle_upsample
        blobs = walk(L, image, oracle_conv(params), want=list(graphs.NANODET_OUTPUTS), upsample_fn=oracle_upsample)
        return oracle_detect([blobs[b] for b in graphs.NANODET_OUTPUTS], [8, 16, 32, 64])

    yield net, x, want
    net.close()


def test_every_call_decodes_its_own_image(detector):
    from graph_support import assert_same_detections
    net, x, want = detector
    rng, counts = np.random.default_rng(7), set()
    for call in range(5):
        image = x if call == 0 else np.clip(x + rng.uniform(-0.2, 0.2, size=x.shape), 0, 1).astype(np.float32)
        rows, count = net.forward_rows("data", image, "nanodet")
        expect = want(image)
        assert count == expect.shape[0], call
        assert_same_detections(rows, expect)
        counts.add(rows.tobytes())
    assert len(counts) == 5  # the images do differ


def test_a_wait_that_ran_out_is_an_error_of_the_call(detector):
    net, x, _ = detector
    ctx = net.context()
    for _ in range(3):  # layer by layer at first, replayed later on
        before = net.forward_rows("data", x, "nanodet")
        ctx.check(ctx.lib.ott_set_wait_limit_ms(ctx.h, 5))
        ctx.check(ctx.lib.ott_debug_wait_probe(ctx.h))
        ctx.check(ctx.lib.ott_set_wait_limit_ms(ctx.h, 2000))
        with pytest.raises(RuntimeError, match="gave up a bounded wait"):
            net.forward_rows("data", x, "nanodet")
        after = net.forward_rows("data", x, "nanodet")
        assert after[1] == before[1] and np.array_equal(after[0], before[0])
