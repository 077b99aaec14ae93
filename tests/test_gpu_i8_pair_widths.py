"""The INT8 CTA-pair GEMM at token counts whose tiles are 160, 192, 224 and 256 tokens wide, against cuBLASLt's exact
sums.  Tolerance: none."""

import pytest
import torch

pytestmark = pytest.mark.gpu


# (tokens, channels): one wave of narrow tiles; two; a last tile of one token; whole tiles; the widest
@pytest.mark.parametrize("M,N", [(777, 4096), (777, 6144), (1500, 4096), (1024, 6144), (961, 6144), (1025, 4096), (2048, 4096)])
def test_every_width_matches_exact_sums(M, N):
    from liquidgemm_b200 import ops
    K = 384
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randint(-128, 128, (M, K), device="cuda", dtype=torch.int8, generator=g)
    b = torch.randint(-128, 128, (N, K), device="cuda", dtype=torch.int8, generator=g)
    pad = -M % 32
    acc = torch._int_mm(torch.cat([a, a.new_zeros(pad, K)]), b.t())[:M]
    assert torch.equal(torch.ops.liquidgemm.wgmma_i8_gemm(a, b), acc)
    sa, sb = torch.rand(M, device="cuda", generator=g) * 0.02, torch.rand(N, device="cuda", generator=g) * 0.01
    want = (acc.float() * sa[:, None]) * sb
    for code, dt in ((0, torch.bfloat16), (1, torch.float16), (2, torch.float32)):
        assert torch.equal(torch.ops.liquidgemm.i8_gemm_scaled(a, b, sa, sb, code), want.to(dt))
    ops.poll_status()
