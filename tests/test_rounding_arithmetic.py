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


def _fma(a, b, c):
    """float32 fused multiply-add: the exact sum rounded to odd in float64, then to float32."""
    p, c = a.astype(np.float64) * np.float64(b), c.astype(np.float64)      # 24 x 24 bits: exact
    hi = p + c
    t = hi - p
    err = (p - (hi - t)) + (c - t)
    bits = hi.view(np.int64)
    odd = np.where((err > 0) == (hi > 0), bits | 1, bits - 1)
    return np.where((err != 0) & (bits & 1 == 0), odd, bits).view(np.float64).astype(np.float32)


def test_token_scale_is_the_rounded_quotient():
    """max(amax, 1e-12) / 127 by the residual of the product with fl(1 / 127): every mantissa of a binade, and the ends of
    the range of exponents (above 3e38, infinity and NaN are divided)."""
    inv = np.float32(1) / np.float32(127)
    one = (np.arange(1 << 23, dtype=np.uint32) | np.uint32(0x3F800000)).view(np.float32)
    for scale in (1.0, 2.0 ** -39, 2.0 ** 126):
        a = one[:: 1 if scale == 1.0 else 97] * np.float32(scale)
        a = np.maximum(a[a < np.float32(3e38)], np.float32(1e-12))
        q = a * inv
        r = _fma(q, np.float32(-127), a)
        assert np.array_equal(_fma(r, inv, q), a / np.float32(127)), scale
