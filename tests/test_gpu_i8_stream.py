"""The streaming INT8 GEMM of decode and small mixed batches (through ``i8_gemm_scaled`` and ``wgmma_i8_gemm``) against
exact integer sums and the oracle's scaling.  Tolerance: none."""

import numpy as np
import pytest
import torch

from oracle import lqq_oracle as O
from tests.helpers import assert_bits_equal

pytestmark = pytest.mark.gpu


def _case(M, N, K, seed):
    rng = np.random.default_rng(seed)
    a = rng.integers(-128, 128, (M, K), dtype=np.int8)
    b = rng.integers(-128, 128, (N, K), dtype=np.int8)
    a[0], b[0] = -128, -128                    # the largest sum the types allow
    return a, b, (rng.random(M, dtype=np.float32) * 0.02).astype(np.float32), (rng.random(N, dtype=np.float32) * 0.01).astype(np.float32)


# every token-tile width and its edges; one k-step; K too short to cut; many k-ranges; ragged and tiny N; whole tiles
@pytest.mark.parametrize("M", [1, 15, 16, 17, 32, 33, 64, 65, 128, 129, 255])
@pytest.mark.parametrize("N,K", [(1, 128), (200, 640), (256, 4096), (1000, 2176)])
def test_matches_exact_sums(M, N, K):
    from liquidgemm_b200 import ops
    a, b, sa, sb = _case(M, N, K, M * 7 + N + K)
    acc = (a.astype(np.float64) @ b.astype(np.float64).T).astype(np.int64).astype(np.int32)   # below 2^53: exact
    at, bt = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    assert np.array_equal(torch.ops.liquidgemm.wgmma_i8_gemm(at, bt).cpu().numpy(), acc)
    for code in (0, 1, 2):
        y = torch.ops.liquidgemm.i8_gemm_scaled(at, bt, torch.from_numpy(sa).cuda(), torch.from_numpy(sb).cuda(), code)
        assert_bits_equal(y, O.scale_f32(acc, sa, sb), code, f"{M}x{N}x{K}")
    ops.poll_status()


@pytest.mark.parametrize("M", [4, 100])
def test_more_tiles_than_cta_slots(monkeypatch, M):
    """Whole tiles in more than one wave (the streaming kernel at 4 tokens, the persistent one at 100), the same bits from
    the entry point that takes no workspace, and from the persistent kernel at both."""
    from liquidgemm_b200 import ops
    from liquidgemm_b200._lib import lib, check
    N, K = 40000, 384
    a, b, sa, sb = _case(M, N, K, M)
    acc = (a.astype(np.float64) @ b.astype(np.float64).T).astype(np.int64).astype(np.int32)
    at, bt = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    assert np.array_equal(torch.ops.liquidgemm.wgmma_i8_gemm(at, bt).cpu().numpy(), acc)
    c = torch.empty(M, N, dtype=torch.int32, device="cuda")
    check(lib.lq_i8_gemm_i32(at.data_ptr(), bt.data_ptr(), c.data_ptr(), M, N, K, torch.cuda.current_stream().cuda_stream), "i8")
    assert np.array_equal(c.cpu().numpy(), acc)
    monkeypatch.setenv("LQ_I8_PAIR", "0")
    assert np.array_equal(torch.ops.liquidgemm.wgmma_i8_gemm(at, bt).cpu().numpy(), acc)
    ops.poll_status()
