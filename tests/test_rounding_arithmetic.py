"""The arithmetic of the register quantisers, restated in numpy and compared with the divisions it replaces."""

import numpy as np

MAGIC = np.float32(12582912.0)


def test_code_quotients_need_no_division():
    """Every (q - lo, step) of the 4-bit level: the product with fl(1 / step), rounded to a multiple of 2^-10 by the
    fused addition of 1.5 * 2^13 and then to an integer, equals rint of the float32 quotient (half to even)."""
    d = np.arange(0, 239, dtype=np.float32)
    for step in range(1, 17):
        s = np.float32(step)
        inv = np.float32(1) / s
        # the fused multiply-add rounds once: float64 holds the 8 x 24-bit product and its sum with 12288 exactly
        fused = (d.astype(np.float64) * np.float64(inv) + 12288.0).astype(np.float32)
        got = (fused + (MAGIC - np.float32(12288.0))).view(np.int32) & 0xFF
        assert np.array_equal(got, np.rint(d / s).astype(np.int32)), step


def test_safe_distance_covers_both_roundings():
    """Near every half-integer quotient: where x * fl(1 / scale) keeps 2^-14 from it, both roundings agree."""
    rng = np.random.default_rng(0)
    for _ in range(200):
        scale = np.float32(np.exp(rng.uniform(-30, 30)))
        half = (rng.integers(-127, 127, 4000) + 0.5)
        x = (half * np.float64(scale) * (1 + rng.uniform(-1, 1, 4000) * 2.0 ** rng.integers(-26, -10, 4000))).astype(np.float32)
        inv = np.float32(1) / scale
        prod = x.astype(np.float64) * np.float64(inv)          # exact: 24 x 24 bits
        near = np.rint(prod)
        safe = np.abs(prod - near).astype(np.float32) < np.float32(0.5 - 2.0 ** -14)
        assert np.array_equal(near[safe], np.rint(x / scale)[safe])
        assert safe.any() and not safe.all()
