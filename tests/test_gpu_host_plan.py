"""A recorded step of host-buffer linears (``ops.HostStepPlan``): uploads, linears and downloads on streams of their own,
replayed on changed inputs, against the device path.  Tolerance: none."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_streams", [1, 3, 5])
def test_replays_follow_the_inputs(n_streams):
    from liquidgemm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(n_streams)
    requests, layers = [], []
    # quantising GEMV, decode tensor-core kernel, split tile kernel, pair kernel, no tokens at all
    for m, n, k in [(1, 512, 1024), (2, 40064, 256), (5, 1024, 512), (40, 384, 2048), (300, 4096, 1024), (0, 128, 128), (1, 512, 1024)]:
        qw, blob = ops.quantize_weight_cuda(torch.randn(n, k, device="cuda", generator=g), 64, want_codes=False, want_blob=True)
        layers.append({"s1": qw.s1, "s_u8": qw.s_u8, "offset_a": qw.offset_a, "N": n, "K": k, "rs": blob.reshape(-1)})
        requests.append((torch.zeros(m, k, dtype=torch.float16).pin_memory(), {"s1": qw.s1, "N": n, "K": k, "rs": blob.reshape(-1)},
                         torch.zeros(m, n, dtype=torch.float16).pin_memory()))
    plan = ops.HostStepPlan(requests, n_streams=n_streams)
    for _ in range(3):
        for x, _, _ in requests:
            x.copy_(torch.randn(x.shape, device="cuda", generator=g))
        plan.run()
        plan.synchronize()
        for (x, _, y), layer in zip(requests, layers):
            assert torch.equal(y, ops.w4a8_linear(x.cuda(), layer).cpu()), tuple(y.shape)
    ops.poll_status()


def _layer(n, k, g):
    from liquidgemm_b200 import ops
    qw, blob = ops.quantize_weight_cuda(torch.randn(n, k, device="cuda", generator=g) * 0.05, 64, want_codes=False, want_blob=True)
    return {"s1": qw.s1, "s_u8": qw.s_u8, "offset_a": qw.offset_a, "N": n, "K": k, "rs": blob.reshape(-1)}


def _pinned(m, k):
    return torch.zeros(m, k, dtype=torch.float16).pin_memory()


@pytest.mark.parametrize("n_streams", [1, 3])
def test_requests_that_share_memory_run_in_order(n_streams):
    """One request's output is the next one's input; an input is overwritten by a later output; two requests write the
    same output, the later one last.  Every replay starts from new values."""
    from liquidgemm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(7)
    up, down, again = _layer(2048, 512, g), _layer(512, 2048, g), _layer(2048, 512, g)
    x, mid, end = _pinned(5, 512), _pinned(5, 2048), _pinned(5, 2048)
    # the second request reads what the first wrote and writes over what the first read, and so on through the chain
    requests = [(x, up, mid), (mid, down, x), (x, again, end), (x, up, end), (end, down, x)]
    plan = ops.HostStepPlan(requests, n_streams=n_streams)
    for _ in range(4):
        x.copy_(torch.randn(x.shape, device="cuda", generator=g))
        h = ops.w4a8_linear(x.cuda(), up)
        d = ops.w4a8_linear(h, down)
        last = ops.w4a8_linear(d, up)
        plan.run()
        plan.synchronize()
        assert torch.equal(mid, h.cpu()) and torch.equal(end, last.cpu())
        assert torch.equal(x, ops.w4a8_linear(last, down).cpu())
    ops.poll_status()


def test_construction_leaves_no_scratch_by_stream():
    from liquidgemm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(19)
    kept = {k: t.data_ptr() for d in (ops._HOST_SCRATCH, ops._HOST_PLANES) for k, t in d.items()}
    x, y = torch.randn(40, 2048).half().pin_memory(), _pinned(40, 512)
    L = _layer(512, 2048, g)
    plan = ops.HostStepPlan([(x, L, y)], n_streams=5)
    assert torch.equal(y, ops.w4a8_linear(x.cuda(), L).cpu())     # construction has run the step once
    assert kept == {k: t.data_ptr() for d in (ops._HOST_SCRATCH, ops._HOST_PLANES) for k, t in d.items()}
    del plan


def test_refused_requests():
    from liquidgemm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(17)
    L = _layer(128, 256, g)
    good = (_pinned(2, 256), L, _pinned(2, 128))
    for bad in ((_pinned(2, 128), L, _pinned(2, 128)), (good[0], L, _pinned(3, 128)), (good[0].cuda(), L, good[2]),
                (good[0], L, good[2].float()), (good[0], {**L, "s1": L["s1"].cpu()}, good[2])):
        with pytest.raises(RuntimeError):
            ops.HostStepPlan([good, bad])


def test_plans_own_their_buffers():
    """Plans on streams of their own replay side by side without sharing a reduction workspace, however many there are
    (stream handles are pooled)."""
    from liquidgemm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(11)
    layers = [_layer(1024, 4096, g) for _ in range(4)]
    kept = {k: t.data_ptr() for k, t in ops._WORKSPACES.items()}
    plans = []
    for _ in range(12):
        req = [(torch.randn(1, 4096).half().pin_memory(), L, _pinned(1, 1024)) for L in layers]
        plans.append((ops.HostStepPlan(req), req))
    assert kept == {k: t.data_ptr() for k, t in ops._WORKSPACES.items()}
    owned = [t.data_ptr() for p, _ in plans for t in (*p.tokens, *p.outputs, *p.scratch, *p.zeroed) if t.numel()]
    assert len(set(owned)) == len(owned)
    want = [[ops.w4a8_linear(x.cuda(), L).cpu() for x, L, _ in req] for _, req in plans]
    for _ in range(20):
        for p, _ in plans:
            p.run()
    torch.cuda.synchronize()
    for (_, req), w in zip(plans, want):
        assert all(torch.equal(y, e) for (_, _, y), e in zip(req, w))
    ops.poll_status()


def test_a_dropped_plan_keeps_its_buffers_until_its_replays_end():
    from liquidgemm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(13)
    layers = [_layer(4096, 4096, g) for _ in range(6)]
    req = [(torch.randn(40, 4096).half().pin_memory(), L, _pinned(40, 4096)) for L in layers]
    want = [ops.w4a8_linear(x.cuda(), L).cpu() for x, L, _ in req]
    plan = ops.HostStepPlan(req)
    for _, _, y in req:
        y.zero_()
    main = plan.main
    torch.cuda.synchronize()
    for _ in range(20):
        plan.run()
    del plan
    # blocks of the plan's sizes, filled on the stream they were allocated from
    junk = [torch.full((40, 4096), 99.0, dtype=torch.float16, device="cuda") for _ in range(24)]
    main.synchronize()
    assert all(torch.equal(y, e) for (_, _, y), e in zip(req, want))
    del junk


def test_many_replays_of_a_decode_step():
    """Two decoder layers' linears at four tokens, several streams at once, some thousand replays: every output of every
    replay is compared."""
    from liquidgemm_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(23)
    req, want = [], []
    for n, k in [(6144, 4096), (4096, 4096), (28672, 4096), (4096, 14336)] * 2:
        req.append((torch.randn(4, k).half().pin_memory(), _layer(n, k, g), _pinned(4, n)))
        x8, sx = torch.ops.liquidgemm.quant_per_token(req[-1][0].cuda())
        L = req[-1][1]
        want.append(ops.gemm_fused(x8, L["rs"], sx, L["s1"], n, k, 1, splitk=-1).cpu())
    plan = ops.HostStepPlan(req)
    for i in range(3000):
        plan.run()
        plan.synchronize()
        for (_, _, y), w in zip(req, want):
            assert torch.equal(y.view(torch.int16), w.view(torch.int16)), i
            y.zero_()
    ops.poll_status()
