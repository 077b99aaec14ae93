"""``w4a8_linear`` from activations to outputs in one call: the GEMV that quantises its own tokens, and the two-launch
form behind it, against ``quant_per_token`` followed by the fused operator (both tested against the oracle
elsewhere).  Tolerance: none."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from liquidgemm_b200 import ops as _ops
    return _ops


def _layer(ops, n, k, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randn(n, k, generator=g, device="cuda") * 0.03
    qw, blob = ops.quantize_weight_cuda(w, 64, want_codes=False, want_blob=True)
    return {"s1": qw.s1, "s_u8": qw.s_u8, "offset_a": qw.offset_a, "N": n, "K": k, "rs": blob.reshape(-1)}


def _tokens(m, k, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(m, k, generator=g, device="cuda")
    x[:, 5] *= 20
    x[-1, k - 1] = 30.0      # the largest value of the row in the last k-tile
    if m > 1:
        x[0] = 0.0
    return x.to(dtype)


def _two_calls(x, L, bias, code):
    xq, sc = torch.ops.liquidgemm.quant_per_token(x)
    if bias is None:
        return torch.ops.liquidgemm.w4a8_wgmma_rs_fused(xq, L["rs"], L["s_u8"], L["offset_a"], sc, L["s1"], L["N"], L["K"],
                                                        64, code)
    return torch.ops.liquidgemm.w4a8_linear_bias(xq, L["rs"], sc, L["s1"], bias, L["N"], L["K"], code)


def _one_kernel(x, N, K):
    """Whether the call quantises its tokens inside the GEMV: it then needs no scratch for them."""
    import ctypes
    from liquidgemm_b200._lib import lib, check
    plan = (ctypes.c_size_t * 3)()
    check(lib.lq_linear_plan(x.data_ptr(), x.shape[0], N, K, 0, plan), "linear_plan")
    return plan[0] == 0


# one k-tile; fewer k-tiles than CTAs; cut tiles; ranges longer than K (stream-K over many n-tiles); ragged N; long K
SHAPES = [(64, 128), (192, 256), (1280, 8192), (4096, 4096), (40000, 256), (28672, 1024), (19200, 4096), (1024, 28672)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("N,K", SHAPES)
def test_one_call_equals_two(ops, dtype, N, K):
    L = _layer(ops, N, K, N + K)
    code = {torch.bfloat16: 0, torch.float16: 1, torch.float32: 2}[dtype]
    bias = torch.randn(N, device="cuda").to(dtype)
    for M in (1, 2, 3, 4, 5, 8, 9, 40):
        x = _tokens(M, K, dtype, M)
        want = _two_calls(x, L, None, code)
        assert torch.equal(ops.w4a8_linear(x, L), want), M
        got = torch.ops.liquidgemm.w4a8_linear(x, L["rs"], L["s_u8"], L["offset_a"], L["s1"], bias, N, K, 64, code)
        assert torch.equal(got, _two_calls(x, L, bias, code)), M
        assert _one_kernel(x, N, K) == (M <= 2), M
        if M <= 4:
            buf = torch.empty(x.numel() + 1, dtype=dtype, device="cuda")   # unaligned activations: two launches at any M
            buf[1:] = x.reshape(-1)
            assert not _one_kernel(buf[1:].view(M, K), N, K)
            assert torch.equal(ops.w4a8_linear(buf[1:].view(M, K), L), want), M
    ops.poll_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_special_activations(ops, dtype):
    """One kind of value a row, alone and beside an ordinary row, through the GEMV's own scales and rounding; four such
    rows through the two launches."""
    N, K = 512, 1024
    L = _layer(ops, N, K, 3)
    code = {torch.bfloat16: 0, torch.float16: 1, torch.float32: 2}[dtype]
    bits = torch.int32 if dtype == torch.float32 else torch.int16
    fi = torch.finfo(dtype)
    base = _tokens(9, K, dtype, 1)[1:]
    base[0, 3] = float("nan")
    base[1, 4] = float("inf")
    base[2, 5], base[2, 900] = float("-inf"), float("nan")
    base[3, K - 1] = fi.max
    base[4] = fi.tiny
    base[5] = fi.min
    base[6] = float("nan")
    base[7] = 0.0
    plain = _tokens(2, K, dtype, 2)[1:]
    cases = [row.view(1, K).clone() for row in base] + [torch.cat([row.view(1, K), plain]) for row in base]
    cases += [torch.cat([plain, row.view(1, K)]) for row in base]
    assert all(_one_kernel(x, N, K) for x in cases)
    for x in cases + [base[:4].clone()]:
        got, want = ops.w4a8_linear(x, L), _two_calls(x, L, None, code)
        assert torch.equal(got.view(bits), want.view(bits))


def test_refusals_stay(ops):
    L = _layer(ops, 128, 256, 0)
    good = _tokens(2, 256, torch.float16, 0)
    for bad in (good.cpu(), good[0], good.to(torch.float64), good[:, :128].contiguous()):
        with pytest.raises((RuntimeError, KeyError, NotImplementedError)):
            ops.w4a8_linear(bad, L)
    with pytest.raises(RuntimeError):
        ops.w4a8_linear(good, {**L, "rs": L["rs"][:-1]})
    with pytest.raises(RuntimeError):
        ops.w4a8_linear(good, {**L, "s1": L["s1"][:-1]})
    assert ops.w4a8_linear(good[:0], L).shape == (0, 128)
    assert torch.equal(ops.w4a8_linear(good.t().contiguous().t(), L), ops.w4a8_linear(good, L))


@pytest.mark.parametrize("M", [3, 5, 8, 9, 32, 64])
@pytest.mark.parametrize("shift", [0, 1024, -1024])
def test_outputs_over_the_activations(ops, M, shift):
    """From three tokens on the outputs may lie over the activations (here at the same address, or some elements before or
    behind it): the tokens are quantised into the scratch first."""
    from liquidgemm_b200._lib import lib, check
    N = K = 4096
    L, x = _layer(ops, N, K, 1), _tokens(M, K, torch.bfloat16, M)
    want = _two_calls(x, L, None, 0)
    buf = torch.empty(M * K + 2048, dtype=torch.bfloat16, device="cuda")
    src, dst = buf[1024:1024 + M * K], buf[1024 + shift:1024 + shift + M * N]
    nscratch, nws, kind = ops._linear_sizes(src.data_ptr(), M, N, K, 0)
    scratch = torch.empty(nscratch, dtype=torch.uint8, device="cuda")
    ws = ops._workspace(nws, x.device) if kind != 1 else torch.empty(nws, dtype=torch.uint8, device="cuda")
    for _ in range(20):
        src.copy_(x.view(-1))
        check(lib.lq_w4a8_linear(src.data_ptr(), 0, L["rs"].data_ptr(), L["s1"].data_ptr(), None, dst.data_ptr(), 0, M, N, K, 0,
                                 scratch.data_ptr(), nscratch, None if ws is None else ws.data_ptr(),
                                 0 if ws is None else ws.numel(), torch.cuda.current_stream().cuda_stream), "w4a8_linear")
        assert torch.equal(dst.view(M, N), want)
    ops.poll_status()
