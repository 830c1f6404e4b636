"""GPU: the host-buffer forward replays a captured graph from the third call of a shape on: every call must equal the checker, with
changing inputs and batch sizes, more shapes than are kept, parameters replaced in between, an int8 output blob (which is not
captured), copies longer than the staging ring, pinned buffers, memory refused to a capture, and a Net compiled again."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def small():
    from graph_support import build_net, oracle_conv, oracle_conv_for_calibration
    from graph_walk import calibrate, walk
    from tensor_b200 import graphs
    L = graphs.shufflenetv2_layers(40, 48, batch=1, stage_repeats=(2, 2, 2))
    params = graphs.make_params(L, seed=21)
    calibrate(L, params, np.random.default_rng(0).uniform(0, 1, size=(1, 3, 40, 48)).astype(np.float32), oracle_conv_for_calibration)
    net = build_net(L, params)
    yield net, params, lambda x, blob: walk(L, x, oracle_conv(params), want=[blob])[blob]
    net.close()


def test_every_call_of_a_shape(small):
    net, params, want = small
    rng = np.random.default_rng(1)
    for n in (1, 2, 1, 2, 3, 1, 4, 5, 6, 1, 1, 6):  # six shapes, four of which are kept
        x = rng.uniform(0, 1, size=(n, 3, 40, 48)).astype(np.float32)
        assert np.array_equal(net.forward("data", x, ["conv5"])[0].view(np.int32), want(x, "conv5").view(np.int32)), n


def test_replaced_parameters_take_effect(small):
    net, params, want = small
    x = np.random.default_rng(2).uniform(0, 1, size=(1, 3, 40, 48)).astype(np.float32)
    for _ in range(3):
        before = net.forward("data", x, ["conv5"])[0]
    p = params["conv5"]
    p["bias"] = p["bias"] + np.float32(0.25)
    net.set_conv_params("conv5", p["weight"], p["bias"], p["w_scales"], p["in_scales"], p["out_scales"])
    for _ in range(3):
        after = net.forward("data", x, ["conv5"])[0]
        assert np.array_equal(after.view(np.int32), want(x, "conv5").view(np.int32)) and not np.array_equal(after, before)


def test_int8_blob_and_long_copies(small):
    net, params, want = small
    rng = np.random.default_rng(3)
    for _ in range(3):
        x = rng.uniform(0, 1, size=(1, 3, 40, 48)).astype(np.float32)
        assert np.array_equal(net.forward("data", x, ["s2b0_r_pw1"])[0], want(x, "s2b0_r_pw1"))
    for _ in range(3):
        x = rng.uniform(0, 1, size=(120, 3, 40, 48)).astype(np.float32)  # 2.8 MB up, 2 MB down: more pieces than the ring has
        assert np.array_equal(net.forward("data", x, ["conv5"])[0][[0, 59, 119]].view(np.int32), want(x[[0, 59, 119]], "conv5").view(np.int32))


def test_pinned_buffers(small):
    net, params, want = small
    shape, out_shape = (2, 3, 40, 48), (2,) + net.blob_shape("conv5")[1:]
    buf = [C.c_void_p(), C.c_void_p()]
    for b, s in zip(buf, (shape, out_shape)):
        assert net.lib.ott_host_alloc(int(np.prod(s)) * 4, C.byref(b)) == 0
    x, y = (np.ctypeslib.as_array(C.cast(b, C.POINTER(C.c_float)), shape=s) for b, s in zip(buf, (shape, out_shape)))
    for seed in range(3):
        x[:] = np.random.default_rng(seed).uniform(0, 1, size=shape)
        y[:] = -1
        net.forward_raw("data", buf[0], False, shape, ["conv5"], [buf[1].value])
        assert np.array_equal(y.view(np.int32), want(x, "conv5").view(np.int32))
    for b in buf:
        net.lib.ott_host_free(b)


def test_memory_refused_to_a_capture(small):
    """The n-th allocation of a shape's second call fails (the first is the capture's input buffer, further ones its temporaries): the
    forward is right all the same, and so is every later one."""
    net, params, want = small
    ctx = net.context()
    rng = np.random.default_rng(5)
    for i, nth in enumerate((1, 2, 5, 20, 40)):
        n = 7 + i
        x = rng.uniform(0, 1, size=(n, 3, 40, 48)).astype(np.float32)
        expect = want(x, "conv5").view(np.int32)
        assert np.array_equal(net.forward("data", x, ["conv5"])[0].view(np.int32), expect)
        ctx.check(ctx.lib.ott_debug_fail_alloc_after(ctx.h, nth))
        for _ in range(3):
            assert np.array_equal(net.forward("data", x, ["conv5"])[0].view(np.int32), expect)
        ctx.check(ctx.lib.ott_debug_fail_alloc_after(ctx.h, 0))


def test_a_capture_that_was_refused_memory_is_tried_again(small):
    """Also of a batch in chunks, whose copies overlap its kernels only when it is captured."""
    net, params, want = small
    ctx = net.context()
    for n, chunk, capturing in ((13, 64, 2), (12, 4, 1)):  # the call that captures: the second one, for chunks the first
        x = np.random.default_rng(n).uniform(0, 1, size=(n, 3, 40, 48)).astype(np.float32)
        expect = want(x, "conv5").view(np.int32)
        taken = 0
        for refuse in (False, True):
            net.set_option("host_chunk", chunk)  # forgets all shapes
            for _ in range(capturing - 1):
                net.forward("data", x, ["conv5"])
            before = _allocations(net)
            ctx.check(ctx.lib.ott_debug_fail_alloc_after(ctx.h, taken))  # the last allocation of that call, a temporary of the capture
            assert np.array_equal(net.forward("data", x, ["conv5"])[0].view(np.int32), expect)
            ctx.check(ctx.lib.ott_debug_fail_alloc_after(ctx.h, 0))
            taken = _allocations(net) - before
        assert taken > 0
        for _ in range(10):
            assert np.array_equal(net.forward("data", x, ["conv5"])[0].view(np.int32), expect)
        before = _allocations(net)
        assert np.array_equal(net.forward("data", x, ["conv5"])[0].view(np.int32), expect)
        assert _allocations(net) == before, (n, chunk)
    net.set_option("host_chunk", 64)


def test_an_output_that_does_not_exist_is_refused_on_every_call(small):
    net, params, want = small
    x = np.zeros((1, 3, 40, 48), np.float32)
    out = np.empty(1, np.float32)
    for _ in range(3):
        with pytest.raises(RuntimeError, match="unknown blob"):
            net.forward_raw("data", x.ctypes.data_as(C.c_void_p), False, x.shape, ["conv99"], [out.ctypes.data])


def _allocations(net):
    """Blocks the Net's context has handed out so far: a replayed forward takes none."""
    ctx = net.context()
    m, h, u, c = (C.c_uint64() for _ in range(4))
    ctx.check(ctx.lib.ott_alloc_stats(ctx.h, C.byref(m), C.byref(h), C.byref(u), C.byref(c)))
    return m.value + h.value


def test_a_shape_in_use_stays_captured_among_many_others(small):
    net, params, want = small
    rng = np.random.default_rng(6)
    hot = rng.uniform(0, 1, size=(1, 3, 40, 48)).astype(np.float32)
    expect = want(hot, "conv5").view(np.int32)
    net.set_option("host_chunk", 64)  # forgets all shapes
    for _ in range(2):
        net.forward("data", hot, ["conv5"])
    for n in list(range(2, 20)) + [2, 3, 4, 5, 2, 3, 4, 5, 6, 6]:  # one-off shapes, then more shapes with graphs than are kept
        net.forward("data", np.repeat(hot, n, axis=0), ["conv5"])
        before = _allocations(net)
        assert np.array_equal(net.forward("data", hot, ["conv5"])[0].view(np.int32), expect)
        assert _allocations(net) == before, n


def test_a_net_compiled_again_forgets_its_graphs():
    from graph_support import build_net, oracle_conv_for_calibration
    from graph_walk import calibrate
    from tensor_b200 import graphs
    L = graphs.shufflenetv2_layers(40, 48, batch=1, stage_repeats=(2, 2, 2))
    params = graphs.make_params(L, seed=22)
    x = np.random.default_rng(0).uniform(0, 1, size=(1, 3, 40, 48)).astype(np.float32)
    calibrate(L, params, x, oracle_conv_for_calibration)
    net, fresh = build_net(L, params), build_net(L, {})
    for _ in range(3):
        before = net.forward("data", x, ["conv5"])[0]
    net.compile()  # the new layers have no parameters yet
    after = net.forward("data", x, ["conv5"])[0]
    assert np.array_equal(after, fresh.forward("data", x, ["conv5"])[0]) and not np.array_equal(after, before)
    net.close()
    fresh.close()


def test_a_graph_file_loaded_into_a_net_forgets_its_graphs(tmp_path):
    """Loading appends the file's layers and makes every layer anew, the ones that have been captured before included."""
    from graph_support import build_net, oracle_conv_for_calibration
    from graph_walk import calibrate
    from tensor_b200 import graphs
    L = graphs.shufflenetv2_layers(40, 48, batch=1, stage_repeats=(2, 2, 2))
    params = graphs.make_params(L, seed=23)
    x = np.random.default_rng(0).uniform(0, 1, size=(1, 3, 40, 48)).astype(np.float32)
    calibrate(L, params, x, oracle_conv_for_calibration)
    path = tmp_path / "more.otter"
    path.write_text(graphs.to_otter_text([dict(type="Input", name="more", output="more", batchsize=1, channel=3, height=8, width=8)]))
    net, fresh = build_net(L, params), build_net(L, {})
    for _ in range(3):
        before = net.forward("data", x, ["conv5"])[0]
    net.load_otter(path)
    after = net.forward("data", x, ["conv5"])[0]
    assert np.array_equal(after, fresh.forward("data", x, ["conv5"])[0]) and not np.array_equal(after, before)
    net.close()
    fresh.close()
