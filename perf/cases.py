"""The work this package does for its users, as cases that can be timed and compared.

Every case goes through the public entry points on the shapes of this repository's benchmark and tests: the four
linears of a Llama-3.1-8B decoder layer, the same four of a Llama-3-70B layer sharded over eight GPUs, and single
matrices of odd sizes.  Kinds of work:

* ``w4``    the W4A8 linear of the serving plugin's 4-bit mode (``ops.w4a8_linear``; with a bias the two operators
            the plugin calls for it), either recorded once in a CUDA graph and replayed, as a serving engine
            does for its decode and small mixed batches, or called eagerly, as it does for prefill;
* ``int8``  the plugin's INT8-weights mode: token quantiser, then the scaled INT8 GEMM;
* ``host``  a decode step whose activations and outputs live in pinned host memory (``ops.HostStepPlan``);
* ``load``  quantising and packing one weight matrix when a model is loaded.

Results are defined bit for bit (exact integer sums, two rounded float32 multiplies, one rounding to the output
type), so outputs are compared exactly.
"""

import torch

from liquidgemm_b200 import ops

GROUP = 64

# (out features, in features) of the linears of one decoder layer
LAYERS = {
    "8b": ((6144, 4096), (4096, 4096), (28672, 4096), (4096, 14336)),
    "70b_tp8": ((1280, 8192), (1024, 8192), (7168, 8192), (1024, 28672)),
}
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
CODES = {"bf16": 0, "fp16": 1, "fp32": 2}


def listed():
    return [
        # The smallest call: one attention output projection for one token, called eagerly from Python, where the
        # host path and the launches count.
        dict(name="single_m1_eager", kind="w4", shapes="4096x4096", layers=1, M=1, dtype="bf16", bias=False, graph=False),
        # One user's decode step (four decoder layers of it).
        dict(name="decode_m1", kind="w4", shapes="8b", layers=4, M=1, dtype="bf16", bias=False, graph=True),
        # A small serving batch.
        dict(name="decode_m16", kind="w4", shapes="8b", layers=4, M=16, dtype="fp16", bias=False, graph=True),
        # A large decode batch on a model whose linears have biases.
        dict(name="decode_m64_bias", kind="w4", shapes="8b", layers=4, M=64, dtype="bf16", bias=True, graph=True),
        # One rank's share of a large model, sharded eight ways along the output channels: small, long-K matrices.
        dict(name="decode_tp8_m8", kind="w4", shapes="70b_tp8", layers=4, M=8, dtype="bf16", bias=False, graph=True),
        # Decode in the plugin's INT8-weights mode.
        dict(name="decode_int8_m8", kind="int8", shapes="8b", layers=2, M=8, dtype="bf16", bias=False, graph=True),
        # A decode step driven from host buffers, copies included.
        dict(name="host_step_m4", kind="host", shapes="8b", layers=2, M=4, dtype="fp16", bias=False, graph=True),
        # A mixed batch: a short prompt beside running decodes, no multiple of any tile.
        dict(name="mixed_m333", kind="w4", shapes="8b", layers=2, M=333, dtype="bf16", bias=False, graph=True),
        # Prefill of one prompt of ordinary length, and a long one.
        dict(name="prefill_m2048", kind="w4", shapes="8b", layers=1, M=2048, dtype="fp16", bias=False, graph=False),
        dict(name="prefill_m8192", kind="w4", shapes="8b", layers=1, M=8192, dtype="bf16", bias=False, graph=False),
        # Prefill of a ragged length in INT8-weights mode.
        dict(name="prefill_int8_m1500", kind="int8", shapes="8b", layers=1, M=1500, dtype="bf16", bias=False, graph=False),
        # Model load: quantise and pack the widest matrix of a layer.
        dict(name="load_gate_up", kind="load", shapes="28672x4096", layers=1, M=0, dtype="bf16", bias=False, graph=False),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choices(["w4_graph", "w4_eager", "int8_graph", "int8_eager", "host", "load"], [40, 20, 12, 12, 8, 8])[0]
    dtype = rng.choices(["bf16", "fp16", "fp32"], [55, 35, 10])[0]
    odd = "%dx%d" % (64 * _log_uniform(rng, 4, 448), 128 * _log_uniform(rng, 4, 112))
    shapes = rng.choice(["8b", "70b_tp8", odd])
    case = dict(kind=kind.split("_")[0], shapes=shapes, layers=1, M=0, dtype=dtype, bias=False, graph=kind.endswith("graph"))
    if kind == "load":
        case["shapes"] = odd
    elif kind == "host":
        case.update(M=_log_uniform(rng, 1, 64), dtype=rng.choice(["bf16", "fp16"]), graph=True)
    else:
        case.update(M=_log_uniform(rng, 1, 512) if case["graph"] else _log_uniform(rng, 1, 6000),
                    bias=case["kind"] == "w4" and rng.random() < 0.25)
        if case["graph"] and case["M"] <= 64:
            case["layers"] = 2
    return case


def _matrices(case):
    one = LAYERS.get(case["shapes"]) or (tuple(int(v) for v in case["shapes"].split("x")),)
    return one * case["layers"]


def _weight(n, k, dtype, gen):
    """Gaussian weights with one entry in a thousand twenty times larger."""
    w = torch.randn(n, k, device="cuda", dtype=torch.float32, generator=gen).mul_(0.02)
    w.mul_(torch.where(torch.rand(n, k, device="cuda", generator=gen) < 1e-3, 20.0, 1.0))
    return w.to(dtype)


def _activations(m, k, dtype, gen):
    """Gaussian activations with one channel in a hundred ten times larger."""
    hot = torch.where(torch.rand(k, device="cuda", generator=gen) < 0.01, 10.0, 1.0)
    return (torch.randn(m, k, device="cuda", generator=gen) * hot).to(dtype)


def _w4_layer(w):
    qw, blob = ops.quantize_weight_cuda(w, GROUP, want_codes=False, want_blob=True)
    return {"s1": qw.s1, "s_u8": qw.s_u8, "offset_a": qw.offset_a, "N": qw.N, "K": qw.K, "rs": blob.reshape(-1)}


def _int8_layer(w):
    qw, _ = ops.quantize_weight_cuda(w, GROUP, want_codes=True, want_blob=False)
    w8 = torch.ops.liquidgemm.dequant_weight(qw.qweight_u4, qw.s_u8, qw.offset_a, qw.N, qw.K, GROUP)
    return {"s1": qw.s1.view(-1, 1), "w8": w8}


def _forward(state):
    """Every linear of the case once, on its own activations."""
    kind, code, out = state["kind"], state["code"], []
    for layer, x, bias in zip(state["weights"], state["x"], state["bias"]):
        if kind == "int8":
            x8, ascale = torch.ops.liquidgemm.quant_per_token(x)
            out.append(torch.ops.liquidgemm.i8_gemm_scaled(x8, layer["w8"], ascale, layer["s1"], code))
        elif bias is None:
            out.append(ops.w4a8_linear(x, layer))
        else:
            x8, ascale = torch.ops.liquidgemm.quant_per_token(x)
            out.append(torch.ops.liquidgemm.w4a8_linear_bias(x8, layer["rs"], ascale, layer["s1"], bias, layer["N"],
                                                             layer["K"], code))
    return out


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    dtype = DTYPES[case["dtype"]]
    mats = _matrices(case)
    state = {"kind": case["kind"], "code": CODES[case["dtype"]]}
    if case["kind"] == "load":
        state["w"] = _weight(*mats[0], dtype, gen)
        return state
    make = _int8_layer if case["kind"] == "int8" else _w4_layer
    state["weights"] = [make(_weight(n, k, torch.bfloat16, gen)) for n, k in mats]
    state["x"] = [_activations(case["M"], k, dtype, gen) for _, k in mats]
    state["bias"] = [(torch.randn(n, device="cuda", generator=gen) * 0.1).to(dtype) if case["bias"] else None for n, _ in mats]
    if case["kind"] == "host":
        y = [torch.empty((case["M"], n), dtype=dtype, pin_memory=True) for n, _ in mats]
        x = [t.cpu().pin_memory() for t in state.pop("x")]
        state["plan"] = ops.HostStepPlan(list(zip(x, state["weights"], y)))
        state["y"] = y
    elif case["graph"]:
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            _forward(state)
            stream.synchronize()
            state["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(state["graph"], stream=stream):
                state["y"] = _forward(state)
        torch.cuda.current_stream().wait_stream(stream)
    return state


def run(state):
    if "plan" in state:
        state["plan"].run()
        state["plan"].synchronize()   # a host-driven loop reads the outputs next
        return state["y"]
    if "graph" in state:
        state["graph"].replay()
        return state["y"]
    if state["kind"] == "load":
        qw, blob = ops.quantize_weight_cuda(state["w"], GROUP, want_codes=False, want_blob=True)
        return [qw.s1, qw.s_u8, qw.offset_a, blob]
    return _forward(state)


def work(case):
    size = torch.finfo(DTYPES[case["dtype"]]).bits // 8
    nbytes = flops = 0
    for n, k in _matrices(case):
        params = 2 * n * (k // GROUP) + 4 * n
        if case["kind"] == "load":
            # read the weight; write the codes with their steps and offsets, and the steps, offsets and scales again
            nbytes += n * k * size + n * k // 2 + 2 * n * (k // GROUP) + params
            flops += 4 * n * k
            continue
        weights = n * k + 4 * n if case["kind"] == "int8" else n * k // 2 + params
        nbytes += weights + case["M"] * (n + k) * size + (n * size if case["bias"] else 0)
        flops += 2 * case["M"] * n * k
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # integer sums are exact in any order and the rounding steps of the epilogue are defined one by one
    return "exact"
