"""The kernels write both int8 rounding rules as trunc(v + copysign(h, v)) in fp32: h = 0.5 is the packed rule as it stands, and with
h = 0.5 - 2^-25 the same sum rounds half away from zero. Here against the rule itself, around every half up to 300, at the ends of
binades, and on random bit patterns up to 2^23 in magnitude."""
import numpy as np


def test_half_away_as_a_constant():
    h = np.float32(0.5) - np.float32(2.0 ** -25)
    assert h == np.nextafter(np.float32(0.5), np.float32(0))
    halves = (np.arange(0, 600, dtype=np.float32) / 2)[:, None].view(np.int32) + np.arange(-200, 201, dtype=np.int32)[None, :]
    binades = (np.arange(0, 151, dtype=np.int32)[:, None] << 23) + np.arange(-200, 201, dtype=np.int32)[None, :]
    random = np.random.default_rng(0).integers(0, 0x4B000000, 8_000_000, dtype=np.int64).astype(np.int32)
    bits = np.concatenate([halves.reshape(-1), binades.reshape(-1), random])
    v = bits[(bits >= 0) & (bits < 0x4B000000)].view(np.float32)
    got = np.trunc(v + h)  # fp32 sums
    exact = np.floor(v.astype(np.float64) + 0.5)
    assert got.dtype == np.float32 and np.array_equal(got.astype(np.float64), exact)
    assert np.array_equal(np.trunc(-v - h), -got)  # the other sign mirrors it
