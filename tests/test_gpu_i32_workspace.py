"""int32 accumulators at a token count whose scaled call takes the GEMV: both use the same all-zero reduction buffer, and
each leaves it all zero."""

import numpy as np
import pytest
import torch

from oracle import lqq_oracle as O
from tests.helpers import assert_bits_equal, random_lqq, random_tokens, to_torch_qw

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 256, 28672), (2, 4096, 14336), (1, 28672, 4096), (3, 24000, 512), (4, 256, 28672), (2, 203, 28672)])
def test_buffer_stays_zero(M, N, K):
    from liquidgemm_b200 import ops
    from liquidgemm_b200._lib import lib
    # the scaled call takes the GEMV, like one token (at three and four: too many tiles, or too long a k-range, for the decode kernel)
    assert lib.lq_gemm_workspace_kind(M, N, K, 0) == 2 and lib.lq_decode_grid(M, N, K) == lib.lq_decode_grid(1, N, K)
    qw = random_lqq(N, K, seed=M + N)
    tq = to_torch_qw(qw)
    blob = ops._repack_device(tq.qweight_u4, 0, tq.s_u8, tq.offset_a, N, K, 64).reshape(-1)
    x, sc = random_tokens(M, K, seed=M)
    xt, st = torch.from_numpy(x).cuda(), torch.from_numpy(sc).cuda()
    w = (qw.qweight_u4.astype(np.int32) * np.repeat(qw.s_u8, 64, 1) + np.repeat(qw.offset_a, 64, 1).astype(np.int32) - 128)
    acc = (x.astype(np.float64) @ w.astype(np.float64).T).astype(np.int64).astype(np.int32)   # below 2^53: exact
    for _ in range(2):
        assert np.array_equal(ops.gemm_i32(xt, blob, N, K).cpu().numpy(), acc)
        assert_bits_equal(ops.gemm_fused(xt, blob, st, tq.s1, N, K, 0), O.scale_f32(acc, sc, qw.s1), 0, f"{M}x{N}x{K}")
    assert ops._WORKSPACES and all(int(ws.max()) == 0 for ws in ops._WORKSPACES.values())
    ops.poll_status()


@pytest.mark.parametrize("M", [9, 13, 16])
@pytest.mark.parametrize("N,K", [(6144, 4096), (4096, 7680), (4998, 4096)])
def test_scaled_planes_are_cleared(M, N, K):
    """int8 tokens on shapes whose k-ranges are too long for the decode kernel: callers bring the all-zero buffer, the tile
    kernel writes its planes into it, the finish pass clears them; too small a buffer stays refused."""
    from liquidgemm_b200 import ops
    from liquidgemm_b200._lib import lib
    assert lib.lq_gemm_workspace_kind(M, N, K, 0) == 2 and lib.lq_gemm_launches(M, N, K, 0) == 2
    qw = random_lqq(N, K, seed=M + N)
    tq = to_torch_qw(qw)
    blob = ops._repack_device(tq.qweight_u4, 0, tq.s_u8, tq.offset_a, N, K, 64).reshape(-1)
    x, sc = random_tokens(M, K, seed=M)
    xt, st = torch.from_numpy(x).cuda(), torch.from_numpy(sc).cuda()
    want = ops.gemm_fused(xt, blob, st, tq.s1, N, K, 0, splitk=-1)
    bias = torch.randn(N, device="cuda").to(torch.bfloat16)
    for _ in range(3):
        assert torch.equal(ops.gemm_fused(xt, blob, st, tq.s1, N, K, 0), want)
        assert torch.equal(ops.linear_bias(xt, blob, st, tq.s1, bias, N, K, 0), want + bias)
        assert torch.equal(ops.gemm_i32(xt, blob, N, K), ops.gemm_i32(xt, blob, N, K, splitk=1))
    assert ops._WORKSPACES and all(int(ws.max()) == 0 for ws in ops._WORKSPACES.values())
    y, nb = torch.empty_like(want), lib.lq_gemm_workspace_bytes(M, N, K, 0)
    ws = torch.zeros(nb, dtype=torch.uint8, device="cuda")
    assert lib.lq_w4a8_gemm_fused(xt.data_ptr(), blob.data_ptr(), st.data_ptr(), tq.s1.data_ptr(), y.data_ptr(), 0, M, N, K, 0,
                                  ws.data_ptr(), nb - 1, None) == -3
    ops.poll_status()
