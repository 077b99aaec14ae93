"""Scratch that a kernel could not address is refused by the C entry points before anything reaches a device."""

from liquidgemm_b200._lib import lib

WORKSPACE = -3
BIG = 1 << 40


def test_unaligned_int8_workspace():
    M, N, K = 8, 4096, 4096
    assert 0 < lib.lq_i8_workspace_bytes(M, N, K) < BIG
    for off in (1, 2, 3):
        assert lib.lq_i8_gemm_i32_ws(256, 256, 256, M, N, K, 4096 + off, BIG, None) == WORKSPACE
        assert lib.lq_i8_gemm_scaled_ws(256, 256, 256, 256, 256, 0, M, N, K, 4096 + off, BIG, None) == WORKSPACE


def test_unaligned_or_short_linear_scratch():
    for scratch, nbytes in ((None, BIG), (4096 + 8, BIG), (4096, 8 * 4096)):
        assert lib.lq_w4a8_linear(256, 0, 256, 256, None, 256, 0, 8, 4096, 4096, 0, scratch, nbytes, 4096, BIG, None) == WORKSPACE
