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
