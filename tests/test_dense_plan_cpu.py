"""Which launch a dense layer takes, on the CPU over thousands of layers: narrow weight panels must not cost a launch what the wide ones
would have had (one tile per CTA, one pass over fp32 input), a stride-2 layer takes the form that suits its map, and of the layers with one int8
output only those whose panels waste little have channels as rows."""
import ctypes as C
import random

import pytest

SMS = 148


@pytest.fixture(scope="module")
def plan():
    from tensor_b200 import capi
    lib = capi.library()

    def ask(cin, cout, k, stride, n, h, w, f32):
        out = (C.c_int * 8)()
        assert lib.ott_debug_dense_plan(cin, cout, k, stride, n, h, w, f32, SMS, out) == 0
        return dict(zip(("tiles", "panels", "columns", "per_sm", "inside", "compact", "rows", "halo"), out))

    return ask


def _layers(count, seed):
    rng = random.Random(seed)
    for _ in range(count):
        k = rng.choice((1, 3))
        top = 1024 if k == 1 else 256
        yield (rng.randint(24, top), rng.randint(24, top), k, rng.choice((1, 1, 2)) if k == 3 else 1, rng.randint(1, 64), rng.randint(7, 80), rng.randint(7, 80))


def test_launches_keep_to_the_wave_they_were_planned_for(plan):
    seen = set()
    for layer in _layers(4000, 1):
        for f32 in (0, 1):
            p = plan(*layer, f32)
            ctas = p["tiles"] * p["panels"]
            if p["inside"]:
                # one CTA per SM: a second panel means one more pass over the input, and pays only for a launch of one tile per CTA
                assert f32 and (p["panels"] == 1 or ctas <= SMS), (layer, p)
            if p["compact"]:
                assert ctas <= SMS and (p["inside"] or p["columns"] <= 64), (layer, p)
            else:
                assert p["rows"] == 128
            seen.add((p["inside"], p["compact"], p["columns"] <= 32, p["panels"] > 1))
    assert len(seen) >= 8


@pytest.mark.parametrize("layer,f32,panels,inside", [
    ((205, 56, 1, 1, 20, 47, 18), 0, 1, 0),   # 133 tiles: two panels of 32 would be 266 CTAs that read every activation twice
    ((94, 192, 1, 1, 6, 31, 26), 0, 3, 0),    # 38 tiles: panels of 64, not 228 CTAs of 32
    ((96, 512, 1, 1, 40, 8, 16), 0, 4, 0),    # 40 tiles
    ((232, 232, 1, 1, 1, 10, 10), 0, 8, 0),   # 1 tile: as narrow as it gets
    ((202, 130, 3, 1, 12, 10, 15), 0, 3, 0),  # 24 tiles of a weight-heavy layer: 72 CTAs, not 120
    ((256, 512, 1, 1, 128, 28, 28), 1, 2, 0),
    ((116, 116, 1, 1, 256, 20, 20), 1, 1, 1),
    ((64, 64, 3, 1, 1, 56, 56), 1, 2, 1),
    ((128, 128, 3, 1, 8, 28, 28), 1, 1, 0)])
def test_named_launches(plan, layer, f32, panels, inside):
    p = plan(*layer, f32)
    assert (p["panels"], p["inside"]) == (panels, inside), p


def test_fp32_input_is_not_quantized_once_per_narrow_panel(plan):
    for layer, most in (((196, 140, 1, 1, 5, 48, 31), 2), ((113, 197, 1, 1, 11, 23, 12), 4)):
        p = plan(*layer, 1)
        assert p["panels"] <= most and p["tiles"] * p["panels"] <= SMS, p


def test_stride_two_form_follows_the_map(plan):
    assert plan(64, 128, 3, 2, 32, 75, 75, 0)["halo"] == 2
    assert plan(64, 64, 3, 2, 1, 56, 56, 0)["halo"] == 2
    for flat, tiles in (((53, 44, 3, 2, 101, 9, 59), 202), ((32, 32, 3, 2, 128, 8, 40), 128), ((154, 140, 3, 2, 78, 13, 32), 78)):
        p = plan(*flat, 0)  # twice to three times the tiles as halo tiles of 8 x 16
        assert (p["halo"], p["tiles"]) == (0, tiles), p


@pytest.fixture(scope="module")
def launch():
    from tensor_b200 import capi
    lib = capi.library()

    def ask(cin, cout, k, stride, n, h, w, f32, int8):
        out = (C.c_int * 9)()
        assert lib.ott_debug_dense_launch(cin, cout, k, stride, n, h, w, f32, int8, SMS, out) == 0
        return dict(zip(("tiles", "panels", "columns", "per_sm", "inside", "compact", "rows", "halo", "channel_rows"), out))

    return ask


def test_int8_launches(plan, launch):
    seen = set()
    for layer in _layers(4000, 2):
        cin, cout, k, stride, n, h, w = layer
        for f32 in (0, 1):
            base, p = plan(*layer, f32), launch(*layer, f32, 1)
            without = launch(*layer, f32, 0)
            assert without.pop("channel_rows") == 0 and without == base
            if not p["channel_rows"]:
                assert {key: p[key] for key in base} == base
                continue
            cout_pad, k_total = (cout + 15) // 16 * 16, (cin + 31) // 32 * 32
            assert k == 1 and not p["compact"] and p["halo"] == 0, (layer, p)
            if p["inside"]:  # the input quantized once, in front of all the channels
                assert f32 and p["channel_rows"] == p["rows"] == 64 and p["panels"] == 1 and 4 * cin * n * h * w >= 96 << 20 and h * w % 4 == 0, (layer, p)
                assert cout_pad <= p["columns"] <= 512 and 8 * h * w >= 7 * ((h * w + 63) // 64 * 64) and k_total <= 640, (layer, p)
            else:
                assert p["channel_rows"] == 128 and p["columns"] in (64, 128, 192, 256) and k_total <= 512 + 128, (layer, p)
                last = cout_pad - (p["panels"] - 1) * p["columns"]
                computed = sum((min(p["columns"], c) + 63) // 64 * 64 for c in [p["columns"]] * (p["panels"] - 1) + [last])
                assert computed <= 1.4 * cout_pad, (layer, p)
            seen.add((p["inside"], p["columns"] if not p["inside"] else 0, p["panels"] > 1, p["per_sm"]))
    assert len(seen) >= 8, seen


@pytest.mark.parametrize("layer,f32,panels,columns,inside,rows", [
    ((256, 512, 1, 1, 128, 28, 28), 1, 1, 512, 1, 64),
    ((256, 512, 1, 1, 128, 28, 27), 1, 2, 256, 0, 128),  # 99.1 MB of input
    ((256, 512, 1, 1, 128, 28, 28), 0, 2, 256, 0, 128),
    ((170, 468, 1, 1, 4057, 8, 6), 1, 2, 256, 0, 128),   # tiles of 64 pixels that 48 of an image fill
    ((43, 263, 1, 1, 143215, 2, 2), 1, 2, 160, 0, 0),
    ((700, 47, 1, 1, 42, 44, 80), 1, 1, 48, 1, 0),       # two stages of 768 channels
    ((92, 145, 1, 1, 359, 31, 100), 1, 1, 160, 1, 0),    # three accumulators, one of them 17 channels
    ((434, 37, 1, 1, 27, 54, 70), 1, 1, 64, 1, 64),
    ((64, 256, 1, 1, 128, 56, 56), 0, 1, 256, 0, 128),
    ((58, 58, 1, 1, 64, 40, 40), 0, 1, 64, 0, 128),
    ((600, 256, 1, 1, 128, 28, 28), 0, 1, 256, 0, 0),    # the MMAs are the longer half
    ((64, 64, 3, 1, 256, 56, 56), 0, 1, 64, 0, 0)])
def test_named_int8_launches(launch, layer, f32, panels, columns, inside, rows):
    p = launch(*layer, f32, 1)
    assert (p["panels"], p["columns"], p["inside"], p["channel_rows"]) == (panels, columns, inside, rows), p
