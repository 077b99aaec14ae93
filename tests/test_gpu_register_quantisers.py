"""The quantisers that hold a row in registers (tokens: ``quant_per_token``; weights: ``quantize_weight_cuda``) against
the oracle and, bit for bit on every kind of value, against the general kernels, which an unaligned copy of the same
data still takes.  Tolerance: none."""

import numpy as np
import pytest
import torch

from oracle import lqq_oracle as O

pytestmark = pytest.mark.gpu

DTYPES = [torch.bfloat16, torch.float16, torch.float32]


@pytest.fixture(scope="module")
def ops():
    from liquidgemm_b200 import ops as _ops
    return _ops


def _unaligned(t: torch.Tensor) -> torch.Tensor:
    """A contiguous copy whose data starts one element past a 16-byte boundary."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    buf[1:] = t.reshape(-1)
    out = buf[1:].view(t.shape)
    assert out.is_contiguous() and out.data_ptr() % 16
    return out


def _ragged(rows, k, dtype, seed, denominator):
    """Gaussian rows with outliers, and rows made of near-half-integer multiples of their own scale."""
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(rows, k, generator=g)
    x[:, ::97] *= 10
    if rows > 2:
        x[1] = 0.0
        half = torch.randint(0, int(denominator), (k,), generator=g).float() + 0.5
        half[0] = denominator
        x[2] = half * 0.0371 * (1 + (torch.rand(k, generator=g) - 0.5) * 2.0 ** -21)
    return x.to(dtype)


def _specials(x):
    """Infinities, NaN, the type's extremes and tiny values, one kind a row."""
    fi = torch.finfo(x.dtype)
    x = x.clone()
    x[0, 5] = float("nan")
    x[1, 3] = float("inf")
    x[2, 7], x[2, 9] = float("-inf"), float("nan")
    x[3, 0] = fi.max
    x[4] = fi.tiny
    x[5] = fi.min
    return x


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M,K", [(3, 16), (3, 48), (1, 4096), (5, 4112), (3, 8192), (3, 8208), (4, 14336), (3, 28672),
                                 (3, 32768), (3, 65536), (3, 65552)])
def test_tokens_match_the_oracle(ops, dtype, M, K):
    x = _ragged(M, K, dtype, M * 131 + K, 127)
    xq, sc = torch.ops.liquidgemm.quant_per_token(x.cuda())
    e_q, e_s = O.quantize_activation(x.float().numpy())
    assert np.array_equal(sc.cpu().numpy().view(np.uint32), e_s.view(np.uint32))
    assert np.array_equal(xq.cpu().numpy(), e_q)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("K", [16, 1040, 14336])
def test_tokens_of_every_kind_match_the_general_kernel(ops, dtype, K):
    x = _specials(_ragged(6, K, dtype, K, 127)).cuda()
    a, b = torch.ops.liquidgemm.quant_per_token(x), torch.ops.liquidgemm.quant_per_token(_unaligned(x))
    assert torch.equal(a[0], b[0]) and torch.equal(a[1].view(torch.int32), b[1].view(torch.int32))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("group", [64, 128])
@pytest.mark.parametrize("N,K", [(6, 128), (130, 384), (6, 4096), (6, 4224), (6, 14336), (6, 32768), (6, 32896)])
def test_weights_of_every_kind_match_the_general_kernels(ops, dtype, group, N, K):
    w = _ragged(N, K, dtype, N + K, 119)
    for v in (w, _specials(w)):
        v = v.cuda()
        a, ab = ops.quantize_weight_cuda(v, group, want_codes=True, want_blob=True)
        b, bb = ops.quantize_weight_cuda(_unaligned(v), group, want_codes=True, want_blob=True)
        assert torch.equal(a.s1.view(torch.int32), b.s1.view(torch.int32))
        assert torch.equal(a.s_u8, b.s_u8) and torch.equal(a.offset_a, b.offset_a)
        assert torch.equal(a.qweight_u4, b.qweight_u4) and torch.equal(ab, bb)
        only, none = ops.quantize_weight_cuda(v, group, want_codes=True, want_blob=False)
        assert none is None and torch.equal(only.qweight_u4, a.qweight_u4)
    want = O.quantize_weight(w.float().numpy(), group)
    got, _ = ops.quantize_weight_cuda(w.cuda(), group)
    assert np.array_equal(got.qweight_u4.cpu().numpy(), want.qweight_u4)
    assert np.array_equal(got.s_u8.cpu().numpy(), want.s_u8) and np.array_equal(got.offset_a.cpu().numpy(), want.offset_a)
    ops.poll_status()
