"""The decode tensor-core kernel whose k-ranges meet inside a thread-block cluster: int8 tokens against the oracle, and its
quantising form against the token quantiser followed by the same operator.  Tolerance: none (exact integer sums)."""

import numpy as np
import pytest
import torch

from oracle import lqq_oracle as O
from tests.helpers import assert_bits_equal, random_lqq, random_tokens, to_torch_qw, with_bias_f32

pytestmark = pytest.mark.gpu

# k-tiles x k-ranges: one k-tile; fewer k-tiles than operand stages, as many and one more; every cluster size up to eight
# with even and odd ranges; a ring shorter than the range; ragged N; whole tiles up to one per SM; two CTAs per SM
SHAPES = [(128, 128), (64, 896), (200, 1024), (320, 2176), (1000, 1920), (2048, 2048), (3072, 4224), (3840, 3072), (6144, 640),
          (512, 14336), (6144, 4096), (8960, 2048), (9600, 1152), (18944, 512), (18944, 1152), (12800, 2560)]
TOKENS = [3, 8, 9, 16, 17, 32]


@pytest.mark.parametrize("N,K", SHAPES)
def test_int8_tokens_match_the_oracle(N, K):
    from liquidgemm_b200 import ops
    qw = random_lqq(N, K, seed=N + K)
    tq = to_torch_qw(qw)
    blob = ops._repack_device(tq.qweight_u4, 0, tq.s_u8, tq.offset_a, N, K, 64).reshape(-1)
    w = (qw.qweight_u4.astype(np.int32) * np.repeat(qw.s_u8, 64, 1) + np.repeat(qw.offset_a, 64, 1).astype(np.int32) - 128)
    rng = np.random.default_rng(N)
    for M in TOKENS:
        x, sc = random_tokens(M, K, seed=M)
        acc = (x.astype(np.float64) @ w.astype(np.float64).T).astype(np.int64).astype(np.int32)   # below 2^53: exact
        xt, st = torch.from_numpy(x).cuda(), torch.from_numpy(sc).cuda()
        assert np.array_equal(ops.gemm_i32(xt, blob, N, K).cpu().numpy(), acc), M
        y = O.scale_f32(acc, sc, qw.s1)
        for code in (0, 1, 2):
            assert_bits_equal(ops.gemm_fused(xt, blob, st, tq.s1, N, K, code), y, code, f"{M}x{N}x{K}")
        bias = torch.from_numpy(rng.standard_normal(N).astype(np.float32)).cuda().to(torch.bfloat16)
        got = ops.linear_bias(xt, blob, st, tq.s1, bias, N, K, 0)
        assert_bits_equal(got, with_bias_f32(y, bias.cpu().view(torch.int16).numpy().view(np.uint16), 0), 0, f"bias {M}x{N}x{K}")
    ops.poll_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("N,K", SHAPES)
def test_quantising_form_equals_two_launches(N, K, dtype):
    """Maxima in every part of the cluster's k-range, a zero row, infinities, NaN and halves between two integers."""
    from liquidgemm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(N + K)
    qw, blob = ops.quantize_weight_cuda(torch.randn(N, K, generator=g, device="cuda") * 0.03, 64, want_codes=False, want_blob=True)
    L = {"s1": qw.s1, "s_u8": qw.s_u8, "offset_a": qw.offset_a, "N": N, "K": K, "rs": blob.reshape(-1)}
    code = {torch.bfloat16: 0, torch.float16: 1, torch.float32: 2}[dtype]
    raw = torch.int32 if dtype == torch.float32 else torch.int16
    for M in (3, 4, 5, 7, 8):
        x = torch.randn(M, K, generator=g, device="cuda")
        for m in range(M):
            x[m, (m * K) // M] = 9.0 + m
        x[0] = torch.arange(K, device="cuda").remainder(255) / 2 - 63.5   # scale 1/2 exactly: halves everywhere
        x[1] = 0.0
        x[2, K // 2], x[2, 3] = float("inf"), float("nan")
        x = x.to(dtype)
        xq, sc = torch.ops.liquidgemm.quant_per_token(x)
        want = torch.ops.liquidgemm.w4a8_wgmma_rs_fused(xq, L["rs"], L["s_u8"], L["offset_a"], sc, L["s1"], N, K, 64, code) \
            if N % 64 == 0 else ops.gemm_fused(xq, L["rs"], sc, L["s1"], N, K, code)
        bias = torch.randn(N, device="cuda").to(dtype)
        if N % 64 == 0:
            assert torch.equal(ops.w4a8_linear(x, L).view(raw), want.view(raw)), M
        got = torch.ops.liquidgemm.w4a8_linear(x, L["rs"], L["s_u8"], L["offset_a"], L["s1"], bias, N, K, 64, code)
        assert torch.equal(got.view(raw), (want + bias).view(raw)), M
    ops.poll_status()


def test_several_streams_at_once():
    """Six streams replay graphs of this kernel side by side (int8 tokens and the quantising form, k-ranges longer than
    the seven operands unpacked ahead and longer than the ring), beside the GEMV and the tile kernel's planes and finish pass.  A
    thread that handed a ring stage back too early would meet the next tile's bytes.  Every output of every replay is compared, in
    the stream, with the persistent kernel's."""
    from liquidgemm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(5)
    layers = []
    for N, K in [(4096, 4096), (6144, 4096), (2048, 14336), (1024, 7680), (4096, 14336)]:
        qw, blob = ops.quantize_weight_cuda(torch.randn(N, K, generator=g, device="cuda") * 0.03, 64, want_codes=False, want_blob=True)
        layers.append({"s1": qw.s1, "s_u8": qw.s_u8, "offset_a": qw.offset_a, "N": N, "K": K, "rs": blob.reshape(-1)})
    runs = []
    for M in (1, 2, 3, 8, 16, 32):
        cases = []
        for L in layers:
            x = torch.randn(M, L["K"], generator=g, device="cuda", dtype=torch.bfloat16)
            x8, sx = torch.ops.liquidgemm.quant_per_token(x)
            cases.append((L, x, x8, sx, ops.gemm_fused(x8, L["rs"], sx, L["s1"], L["N"], L["K"], 0, splitk=-1)))
        torch.cuda.synchronize()
        stream, wrong = torch.cuda.Stream(), torch.zeros((), dtype=torch.int64, device="cuda")

        def step():
            out = []
            for L, x, x8, sx, want in cases:
                out.append((ops.w4a8_linear(x, L), want))
                out.append((ops.gemm_fused(x8, L["rs"], sx, L["s1"], L["N"], L["K"], 0), want))
            for y, want in out:
                wrong.add_((y.view(torch.int16) != want.view(torch.int16)).sum())
        with torch.cuda.stream(stream):
            step()
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                step()
        runs.append((M, stream, graph, wrong, cases))
    for _ in range(1500):
        for _, stream, graph, *_ in runs:
            with torch.cuda.stream(stream):
                graph.replay()
    torch.cuda.synchronize()
    for M, _, _, wrong, _ in runs:
        assert int(wrong) == 0, M
    ops.poll_status()


@pytest.mark.parametrize("M", [8, 17, 32])
@pytest.mark.parametrize("N,K", [(384, 2048), (200, 7680), (9728, 1024)])   # K cut evenly, unevenly, not at all
def test_several_destinations(M, N, K):
    """The multi-destination form: two wider matrices, then a sequence in which each launch waits for the flags that the
    one before has raised, one count per CTA."""
    from liquidgemm_b200 import ops
    qw = random_lqq(N, K, seed=N + M)
    tq = to_torch_qw(qw)
    blob = ops._repack_device(tq.qweight_u4, 0, tq.s_u8, tq.offset_a, N, K, 64).reshape(-1)
    x, sc = random_tokens(M, K, seed=M)
    xt, st = torch.from_numpy(x).cuda(), torch.from_numpy(sc).cuda()
    want = O.w4a8_matmul(x, sc, qw)
    ld, col = N + 616, 256
    outs = [torch.full((M, ld), -7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    ops.gemm_fused_scatter(xt, blob, st, tq.s1, [o.data_ptr() for o in outs], ld, col, N, K, 0)
    for o in outs:
        assert_bits_equal(o[:, col:col + N].contiguous(), want, 0, "destinations")
        assert bool((o[:, :col] == -7.0).all()) and bool((o[:, col + N:] == -7.0).all())
    grid, flags = ops.decode_grid(M, N, K), torch.zeros(4, dtype=torch.int32, device="cuda")
    outs = [torch.zeros((M, N), dtype=torch.float16, device="cuda") for _ in range(3)]
    for k, o in enumerate(outs):
        ops.gemm_fused_scatter(xt, blob, st, tq.s1, [o.data_ptr()], N, 0, N, K, 1, flag_ptrs=[flags.data_ptr()], flag_index=k,
                               wait_ptr=(flags.data_ptr() + 4 * (k - 1)) if k else None, wait_value=grid if k else 0)
    for o in outs:
        assert_bits_equal(o, want, 1, "flags")
    assert flags.tolist() == [grid] * 3 + [0]
    ops.poll_status()


@pytest.mark.parametrize("M,N,K", [(17, 4096, 4096), (32, 6144, 2048), (24, 9728, 1024), (8, 17408, 4096)])
def test_calls_without_a_workspace(M, N, K):
    """Where callers are told that none is needed, none is asked for, with int8 tokens and with activations."""
    from liquidgemm_b200 import ops
    from liquidgemm_b200._lib import lib, check
    g = torch.Generator(device="cuda").manual_seed(M + N)
    qw, blob = ops.quantize_weight_cuda(torch.randn(N, K, generator=g, device="cuda") * 0.03, 64, want_codes=False, want_blob=True)
    x = torch.randn(M, K, generator=g, device="cuda", dtype=torch.bfloat16)
    x8, sx = torch.ops.liquidgemm.quant_per_token(x)
    want = ops.gemm_fused(x8, blob.reshape(-1), sx, qw.s1, N, K, 0, splitk=-1)
    st = torch.cuda.current_stream().cuda_stream
    y = torch.empty_like(want)
    check(lib.lq_w4a8_gemm_fused(x8.data_ptr(), blob.data_ptr(), sx.data_ptr(), qw.s1.data_ptr(), y.data_ptr(), 0, M, N, K, 0,
                                 None, 0, st), "w4a8_gemm_fused")
    assert torch.equal(y, want)
    y.zero_()
    nscratch, nws, kind = ops._linear_sizes(x.data_ptr(), M, N, K, 0)
    assert nws == kind == 0
    scratch = torch.empty(nscratch, dtype=torch.uint8, device="cuda")
    check(lib.lq_w4a8_linear(x.data_ptr(), 0, blob.data_ptr(), qw.s1.data_ptr(), None, y.data_ptr(), 0, M, N, K, 0,
                             scratch.data_ptr(), nscratch, None, 0, st), "w4a8_linear")
    assert torch.equal(y, want)
    ops.poll_status()


def test_token_scales_over_the_range():
    """The quantising form's own division by 127 against the token quantiser's, over the exponents of float32."""
    from liquidgemm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(9)
    N, K = 64, 128
    qw, blob = ops.quantize_weight_cuda(torch.randn(N, K, generator=g, device="cuda"), 64, want_codes=False, want_blob=True)
    L = {"s1": qw.s1, "s_u8": qw.s_u8, "offset_a": qw.offset_a, "N": N, "K": K, "rs": blob.reshape(-1)}
    for i in range(300):
        x = torch.randn(8, K, generator=g, device="cuda") * torch.exp2(torch.rand(8, 1, generator=g, device="cuda") * 160 - 40)
        if i == 0:
            x[:, 0] = torch.tensor([3e38, 3.1e38, torch.finfo(torch.float32).max, 1e-12, 0.9e-12, 1.1e-12, 0.0, 127.0], device="cuda")
        xq, sc = torch.ops.liquidgemm.quant_per_token(x)
        want = torch.ops.liquidgemm.w4a8_wgmma_rs_fused(xq, L["rs"], L["s_u8"], L["offset_a"], sc, L["s1"], N, K, 64, 2)
        assert torch.equal(ops.w4a8_linear(x, L).view(torch.int32), want.view(torch.int32)), i
    ops.poll_status()
