"""Operands that the kernel directly before has written: the overlapped launches must wait for them.  Exact sums, so the
tolerance is none."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _exact(a, b):
    """a @ b.T in integers: every partial sum is below 2^53."""
    return (a.double() @ b.double().t()).to(torch.int32)


# streaming kernel with K cut, whole tiles in several waves, its widest token tile; the CTA-pair kernel
@pytest.mark.parametrize("M,N,K", [(8, 4096, 4096), (1, 28672, 2048), (33, 40064, 1024), (200, 1024, 4096), (300, 16384, 512)])
@pytest.mark.parametrize("between", [False, True])
def test_int8_weights_quantised_just_before(M, N, K, between):
    """Both operands from ``quant_per_token``, the weights last, or (a second early-triggering kernel between the
    writer and the reader) the tokens last.  The weights' buffer is the same in every pass, with other contents."""
    from liquidgemm_b200 import ops
    from liquidgemm_b200._lib import lib, check
    g = torch.Generator(device="cuda").manual_seed(M + N)
    ws = [torch.randn(N, K, device="cuda", generator=g, dtype=torch.bfloat16) for _ in range(2)]
    x = torch.randn(M, K, device="cuda", generator=g, dtype=torch.bfloat16)
    w8, sw = torch.zeros(N, K, device="cuda", dtype=torch.int8), torch.zeros(N, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    settled = [torch.ops.liquidgemm.quant_per_token(w) for w in ws]
    x8, sx = torch.ops.liquidgemm.quant_per_token(x)
    torch.cuda.synchronize()
    acc = [_exact(x8, q) for q, _ in settled]
    want = [((a.float() * sx[:, None]) * s).to(torch.bfloat16) for a, (_, s) in zip(acc, settled)]
    got = []
    for i in range(12):
        check(lib.lq_quant_per_token(ws[i & 1].data_ptr(), 0, w8.data_ptr(), sw.data_ptr(), N, K, st), "quant_per_token")
        if between:
            x8, sx = torch.ops.liquidgemm.quant_per_token(x)
        if i < 6:
            got.append(torch.ops.liquidgemm.wgmma_i8_gemm(x8, w8))
        else:
            got.append(torch.ops.liquidgemm.i8_gemm_scaled(x8, w8, sx, sw, 0))
    for i, y in enumerate(got):
        assert torch.equal(y, (acc if i < 6 else want)[i & 1]), i
    ops.poll_status()


# CTA-pair kernel (where it serves: LQ_PAIR_ALWAYS), whole and cut last waves; decode tensor-core kernel; tile kernel with
# K cut and with whole tiles in several waves
RETILED = [(2048, 4096, 1024), (700, 28672, 512), (8, 4096, 4096), (40, 1024, 4096), (100, 40064, 512)]


@pytest.mark.parametrize("M,N,K", RETILED)
@pytest.mark.parametrize("op", ["w4a8_wgmma", "w4a8_wgmma_rs"])
def test_weights_retiled_just_before(monkeypatch, M, N, K, op):
    """The operators that take ``pack_nibbles`` weights re-tile them into scratch (the same block of the allocator in
    every pass, with other contents) and multiply at once."""
    from liquidgemm_b200 import ops
    from liquidgemm_b200.pack import pack_nibbles
    monkeypatch.setenv("LQ_PAIR_ALWAYS", "1")
    g = torch.Generator(device="cuda").manual_seed(M + N)
    layers = []
    for _ in range(2):
        qw, _ = ops.quantize_weight_cuda(torch.randn(N, K, device="cuda", generator=g), 64)
        w8 = torch.ops.liquidgemm.dequant_weight(qw.qweight_u4, qw.s_u8, qw.offset_a, N, K, 64)
        layers.append((pack_nibbles(qw.qweight_u4).contiguous(), qw.s_u8, qw.offset_a, w8))
    x = torch.randint(-127, 128, (M, K), device="cuda", dtype=torch.int8, generator=g)
    torch.cuda.synchronize()
    acc = [_exact(x, w8) for *_, w8 in layers]
    for i in range(8):
        w, s, a, _ = layers[i & 1]
        if op == "w4a8_wgmma":
            y = torch.ops.liquidgemm.w4a8_wgmma(x, w, s, a, N, K, 64)
        else:
            y = torch.ops.liquidgemm.w4a8_wgmma_rs(x, w, s, s, a, N, K, 64, False)
        assert torch.equal(y, acc[i & 1]), i
    ops.poll_status()


@pytest.mark.parametrize("M,N,K", [(1, 4096, 4096), (8, 4096, 4096), (8, 28672, 1024), (40, 1024, 4096)])
@pytest.mark.parametrize("writer", ["quantise", "repack", "copy"])
def test_blob_written_just_before(M, N, K, writer):
    """The package's own writers of tile blobs, into the same buffer with changing contents, directly before a fused
    linear that fetches its first tiles ahead of the stream."""
    from liquidgemm_b200 import ops
    from liquidgemm_b200._lib import lib, check
    g = torch.Generator(device="cuda").manual_seed(M + N)
    ws = [torch.randn(N, K, device="cuda", generator=g, dtype=torch.bfloat16) for _ in range(2)]
    settled = [ops.quantize_weight_cuda(w, 64, want_codes=True, want_blob=True) for w in ws]
    x8, sx = torch.ops.liquidgemm.quant_per_token(torch.randn(M, K, device="cuda", generator=g))
    want = []
    for qw, blob in settled:
        torch.cuda.synchronize()
        want.append(ops.gemm_fused(x8, blob.reshape(-1), sx, qw.s1, N, K, 0))
    blob, (s1, s, a) = torch.zeros_like(settled[0][1]), (torch.empty_like(t) for t in (qw.s1, qw.s_u8, qw.offset_a))
    st = torch.cuda.current_stream().cuda_stream
    torch.cuda.synchronize()
    for i in range(8):
        qw = settled[i & 1][0]
        if writer == "quantise":
            check(lib.lq_quantize_weight(ws[i & 1].data_ptr(), 0, N, K, 64, s1.data_ptr(), s.data_ptr(), a.data_ptr(), None,
                                         blob.data_ptr(), st), "quantize_weight")
        elif writer == "copy":   # a blob that the operator itself has to make contiguous
            y = ops.gemm_fused(x8, settled[i & 1][1].reshape(-1).repeat_interleave(2)[::2], sx, qw.s1, N, K, 0)
            assert torch.equal(y, want[i & 1]), i
            continue
        else:
            check(lib.lq_repack_tiles(qw.qweight_u4.data_ptr(), 0, qw.s_u8.data_ptr(), qw.offset_a.data_ptr(),
                                      blob.data_ptr(), N, K, 64, st), "repack_tiles")
        y = ops.gemm_fused(x8, blob.reshape(-1), sx, qw.s1, N, K, 0)
        assert torch.equal(y, want[i & 1]), i
    ops.poll_status()


def _w4_layer(n, k, g):
    from liquidgemm_b200 import ops
    qw, blob = ops.quantize_weight_cuda(torch.randn(n, k, device="cuda", generator=g) * 0.05, 64, want_codes=False, want_blob=True)
    return {"s1": qw.s1, "s_u8": qw.s_u8, "offset_a": qw.offset_a, "N": n, "K": k, "rs": blob.reshape(-1)}


def _linear_into(y, x, layer, code, s1=None, bias=None):
    """``lq_w4a8_linear`` of activations ``x`` into the given buffer, with the sizes that it reports."""
    from liquidgemm_b200 import ops
    from liquidgemm_b200._lib import lib, check
    M, N, K = x.shape[0], layer["N"], layer["K"]
    nscratch, nws, kind = ops._linear_sizes(x.data_ptr(), M, N, K, 0)
    scratch = torch.empty(max(nscratch, 1), dtype=torch.uint8, device="cuda")
    ws = ops._workspace(nws, x.device) if kind == 2 else torch.empty(max(nws, 1), dtype=torch.uint8, device="cuda")
    check(lib.lq_w4a8_linear(x.data_ptr(), {torch.bfloat16: 0, torch.float16: 1, torch.float32: 2}[x.dtype], layer["rs"].data_ptr(),
                             (layer["s1"] if s1 is None else s1).data_ptr(), None if bias is None else bias.data_ptr(),
                             y.data_ptr(), code, M, N, K, 0, scratch.data_ptr(), nscratch,
                             None if ws is None else ws.data_ptr(), 0 if ws is None else ws.numel(),
                             torch.cuda.current_stream().cuda_stream), "w4a8_linear")


@pytest.mark.parametrize("M", [1, 2, 3, 4, 8, 16, 24, 32, 64])
@pytest.mark.parametrize("N,K", [(4096, 4096), (1000, 1920), (18944, 512), (2048, 14336)])
@pytest.mark.parametrize("what", ["bias", "s1", "copies"])
def test_scales_and_bias_written_just_before(M, N, K, what):
    """The channel scales or the bias are the output of the one-token linear directly before (the same buffer in every
    pass, with other contents), or the operator itself makes them contiguous.  At 1 to 8 tokens the operator that takes
    activations has no quantiser launch in between."""
    from liquidgemm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + N)
    layer, writer = _w4_layer(N, K, g), _w4_layer(N, 512, g)
    x = torch.randn(M, K, device="cuda", generator=g, dtype=torch.bfloat16)
    x8, sx = torch.ops.liquidgemm.quant_per_token(x)
    conds = [torch.randn(1, 512, device="cuda", generator=g, dtype=torch.float32) for _ in range(2)]
    code = 2 if what == "s1" else 0
    vec = torch.zeros(1, N, device="cuda", dtype=torch.float32 if code == 2 else torch.bfloat16)
    plain = torch.randn(N, device="cuda", generator=g).to(torch.bfloat16)

    def args(i):
        if what == "copies":
            s1, b = (layer["s1"], plain) if i == 0 else (layer["s1"] * 2, plain + 1)
            return [t.repeat_interleave(2)[::2] for t in (s1, b)]
        return (vec.view(-1), plain) if what == "s1" else (layer["s1"], vec.view(-1))

    def both(i, settle):
        out = []
        for op in range(2):
            s1, b = args(i)
            if what != "copies":
                _linear_into(vec, conds[1 - i], writer, code)   # the other contents, then at once these
                _linear_into(vec, conds[i], writer, code)
            if settle:
                torch.cuda.synchronize()
            if op:
                out.append(torch.ops.liquidgemm.w4a8_linear(x, layer["rs"], layer["s_u8"], layer["offset_a"], s1, b, N, K, 64, 0))
            else:
                out.append(ops.linear_bias(x8, layer["rs"], sx, s1, b, N, K, 0))
        return out
    want = [both(i, True) for i in range(2)]
    assert not torch.equal(want[0][0], want[1][0])
    got = [both(i & 1, False) for i in range(12)]
    for i, ys in enumerate(got):
        for y, w in zip(ys, want[i & 1]):
            assert torch.equal(y.view(torch.int16), w.view(torch.int16)), i
    ops.poll_status()


@pytest.mark.parametrize("M", [1, 2, 3, 5, 8, 16, 32, 64, 200])
@pytest.mark.parametrize("widths", [(2048, 4096), (1024, 14336)])
def test_chains_reuse_every_buffer(M, widths):
    """Eight linears in a graph, each reading what the one before wrote, through two activation buffers and the same
    scratch (tokens, scales, planes): every address is written anew while the next reader is resident already.  New
    contents in every replay, without synchronising in between."""
    g = torch.Generator(device="cuda").manual_seed(M)
    n, k = widths
    down, up = _w4_layer(n, k, g), _w4_layer(k, n, g)
    a, b = (torch.zeros(M, w, device="cuda", dtype=torch.bfloat16) for w in (k, n))

    def chain(settle=False):
        for _ in range(4):
            for y, x, layer in ((b, a, down), (a, b, up)):
                _linear_into(y, x, layer, 0)
                if settle:
                    torch.cuda.synchronize()
    xs = [torch.randn(M, k, device="cuda", generator=g, dtype=torch.bfloat16) for _ in range(5)]
    want = []
    for x in xs:
        a.copy_(x)
        chain(settle=True)
        want.append(a.clone())
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        chain()
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            chain()
        wrong = torch.zeros((), dtype=torch.int64, device="cuda")
        for i in range(200):
            a.copy_(xs[i % 5])
            graph.replay()
            wrong += (a.view(torch.int16) != want[i % 5].view(torch.int16)).sum()
        stream.synchronize()
    assert int(wrong) == 0


@pytest.mark.parametrize("M,N,K", [(8, 4096, 4096), (33, 1024, 14336), (200, 1024, 4096), (300, 16384, 512)])
def test_int8_layers_reuse_every_buffer(M, N, K):
    """The same for the INT8-weights mode: tokens, token scales and planes at the same addresses, layer after layer."""
    from liquidgemm_b200 import ops
    from liquidgemm_b200._lib import lib, check
    g = torch.Generator(device="cuda").manual_seed(M + N)
    w8 = torch.randint(-127, 128, (N, K), device="cuda", dtype=torch.int8, generator=g)
    sw = torch.rand(N, device="cuda", generator=g)
    xs = [torch.randn(M, K, device="cuda", generator=g, dtype=torch.bfloat16) for _ in range(4)]
    want = [torch.ops.liquidgemm.i8_gemm_scaled(q, w8, s, sw, 0) for q, s in (torch.ops.liquidgemm.quant_per_token(x) for x in xs)]
    torch.cuda.synchronize()
    x8, sx = torch.empty(M, K, device="cuda", dtype=torch.int8), torch.empty(M, device="cuda")
    nb = lib.lq_i8_workspace_bytes(M, N, K)
    ws = torch.empty(max(nb, 1), dtype=torch.uint8, device="cuda")
    ys = [torch.empty(M, N, device="cuda", dtype=torch.bfloat16) for _ in xs]
    st = torch.cuda.current_stream().cuda_stream
    wrong = torch.zeros((), dtype=torch.int64, device="cuda")
    for _ in range(50):
        for x, y in zip(xs, ys):
            check(lib.lq_quant_per_token(x.data_ptr(), 0, x8.data_ptr(), sx.data_ptr(), M, K, st), "quant_per_token")
            check(lib.lq_i8_gemm_scaled_ws(x8.data_ptr(), w8.data_ptr(), sx.data_ptr(), sw.data_ptr(), y.data_ptr(), 0, M, N, K,
                                           ws.data_ptr() if nb else None, nb, st), "i8_gemm_scaled")
        for y, w in zip(ys, want):
            wrong += (y.view(torch.int16) != w.view(torch.int16)).sum()
            y.zero_()
    assert int(wrong) == 0
    ops.poll_status()
