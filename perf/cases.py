"""Performance cases of the affine-Q4 projection library: what a program that serves a model through it has it do.

A case is a dict of plain values. `kind` names the public call:

    project   CudaRuntime.matmul_batch_device      projections that share one activation, buffers on the GPU
    mlp       CudaRuntime.mlp_batch_device         down(silu(gate x) * (up x))
    argmax    CudaRuntime.argmax_batch_device      lm_head and the greedy token of every row
    token     DecodeChain.run                      a whole decode token in one launch (SyntheticStack.build_chain)
    host      CudaRuntime.q4_affine_matmul_mapped_batch   host arrays in, host arrays out
    host_mlp  CudaRuntime.q4_affine_mlp_mapped_batch      the same for the MLP

`m` activation rows of `k` inputs, `rows` output rows per projection, `dtype` of the activation, `offsets` the bytes by
which the tensors of successive projections miss a 16-byte boundary (safetensors shards put them anywhere), `residual`
the form that adds to its output. The sizes are those of the benchmark's layer (hidden 5120, intermediate 17408,
vocabulary 248320; Q/K/V, the four DeltaNet inputs, gate/up and down) and generic ones around them.
"""
import torch

from qwen38_metal_b200 import capi
from qwen38_metal_b200.runtime import CudaRuntime, MappedQ4AffineJob
from qwen38_metal_b200.stack import HIDDEN, INTER, LAYER_ROWS, VOCAB, SyntheticStack

SIGMA = 0.02  # standard deviation of the synthetic weights before quantisation


def _project(name, m, k, rows, dtype="bf16", offsets="0", residual=False):
    return {"name": name, "kind": "project", "m": m, "k": k, "rows": rows, "dtype": dtype, "offsets": offsets,
            "residual": residual}


def listed():
    return [
        # the smallest call of a decode step: one output projection
        _project("decode_5120", 1, HIDDEN, "5120"),
        # a decode layer's projections of the hidden vector in one call, every other tensor off a 16-byte boundary
        _project("decode_layer", 1, HIDDEN, ",".join(str(r) for r in LAYER_ROWS), offsets="0,2"),
        # the down projection of a decode step that adds to the residual stream, fp32 activation
        _project("decode_down_residual", 1, INTER, str(HIDDEN), dtype="f32", offsets="2", residual=True),
        # speculative decoding: four draft tokens verified at once, the layer's largest pair
        _project("verify_gate_up_4", 4, HIDDEN, "17408,17408"),
        # eight concurrent requests, fp32 activations (the reference's type), shard with tensors at odd places
        _project("lanes_qkv_8", 8, HIDDEN, "6144,1024,1024", dtype="f32", offsets="2"),
        # 48 concurrent requests: between decode and prompt
        _project("lanes_down_48", 48, INTER, str(HIDDEN)),
        # a short prompt of odd length through the DeltaNet inputs
        _project("prompt_deltanet_333", 333, HIDDEN, "6144,2048,2048,48", dtype="f32", offsets="0,2"),
        # a prompt block of the benchmark's length, the layer's largest pair: the largest call
        _project("prompt_gate_up_2048", 2048, HIDDEN, "17408,17408"),
        # the whole MLP of a prompt block that does not fill its tiles, off a 16-byte boundary
        {"name": "prompt_mlp_1000", "kind": "mlp", "m": 1000, "k": HIDDEN, "inter": INTER, "dtype": "bf16", "offsets": "2"},
        # greedy tokens of four verified positions
        {"name": "verify_argmax_4", "kind": "argmax", "m": 4, "k": HIDDEN, "rows": str(VOCAB), "dtype": "bf16", "offsets": "0"},
        # a decode token through the persistent chain; two layers, so that outputs of different evaluation orders can be
        # compared (the stack amplifies last-bit differences from layer to layer)
        {"name": "token_chain", "kind": "token", "layers": 2, "vocab": VOCAB},
        # host arrays in and out, as the reference's NativeWeights calls it: Q/K/V of one token
        {"name": "host_qkv", "kind": "host", "m": 1, "k": HIDDEN, "rows": "6144,1024,1024", "dtype": "f32", "offsets": "2"},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def _inputs(rng):
    """An input width: mostly the widths of model layers (multiples of 512), else any whole number of groups."""
    step = 512 if rng.random() < 0.75 else 64
    return step * _log_int(rng, max(1, 1024 // step), INTER // step)


def _one(rng):
    kind = rng.choices(("project", "mlp", "argmax", "token", "host", "host_mlp"), (60, 12, 8, 8, 8, 4))[0]
    dtype = rng.choice(("bf16", "bf16", "f32"))
    offsets = rng.choice(("0", "0", "0,2", "2", "8", "6"))
    if kind == "token":
        return {"kind": kind, "layers": rng.randint(1, 3), "vocab": 8 * _log_int(rng, 4096, VOCAB // 8)}
    if kind == "argmax":
        return {"kind": kind, "m": _log_int(rng, 1, 16), "k": _inputs(rng), "rows": str(_log_int(rng, 32000, VOCAB)),
                "dtype": dtype, "offsets": offsets}
    if kind == "mlp":
        return {"kind": kind, "m": _log_int(rng, 1, 2048), "k": _inputs(rng), "inter": 64 * _log_int(rng, 32, INTER // 64),
                "dtype": dtype, "offsets": offsets}
    if kind == "host_mlp":
        return {"kind": kind, "m": _log_int(rng, 1, 64), "k": _inputs(rng), "inter": 64 * _log_int(rng, 32, INTER // 64),
                "dtype": "f32", "offsets": offsets}
    rows = ",".join(str(_log_int(rng, 48, INTER)) for _ in range(rng.randint(1, 4)))
    if kind == "host":
        return {"kind": kind, "m": _log_int(rng, 1, 64), "k": _inputs(rng), "rows": rows, "dtype": "f32", "offsets": offsets}
    # single rows, short batches, mid-size batches, prompts
    lo, hi = rng.choices(((1, 1), (2, 16), (17, 128), (129, 2048)), (30, 25, 15, 30))[0]
    return {"kind": kind, "m": _log_int(rng, lo, hi), "k": _inputs(rng), "rows": rows, "dtype": dtype, "offsets": offsets,
            "residual": rng.random() < 0.2}


def _cost(case):
    w = work(case)
    return w["bytes"] / 6.5e12 + w["flops"] / 1.6e15


def draw(rng):
    """One more case of the same ranges: sizes spread over their logarithm, no larger than the largest listed case."""
    most = max(_cost(c) for c in listed())
    while True:
        case = _one(rng)
        if _cost(case) <= most:
            return case


def _shapes(case):
    """(output rows, inputs) of every projection of a case."""
    if case["kind"] in ("mlp", "host_mlp"):
        return [(case["inter"], case["k"]), (case["inter"], case["k"]), (case["k"], case["inter"])]
    if case["kind"] == "token":
        layer = [(n, HIDDEN) for n in LAYER_ROWS] + [(HIDDEN, INTER)]
        return layer * case["layers"] + [(case["vocab"], HIDDEN)]
    return [(int(n), case["k"]) for n in case["rows"].split(",")]


class State:
    """Weights on the GPU, activations, output buffers and the runtime that owns them."""

    def __init__(self):
        self.rt = CudaRuntime(0)
        self.chain = None

    def __del__(self):
        if self.chain is not None:
            self.chain.close()
        self.rt.close()


def _weights(state, case, seed):
    """The projections of a case, quantised normal weights; a projection's three tensors share its offset."""
    jobs = []
    offsets = [int(o) for o in case["offsets"].split(",")]
    for i, (n, k) in enumerate(_shapes(case)):
        off = offsets[i % len(offsets)]
        if case["kind"] in ("mlp", "host_mlp"):
            off = offsets[i // 2 % len(offsets)]  # gate and up come from one shard
        w = state.rt.alloc_shard(n * (k // 2) + off)
        s = state.rt.alloc_shard(n * (k // 64) * 2 + off)
        b = state.rt.alloc_shard(n * (k // 64) * 2 + off)
        job = MappedQ4AffineJob(w, off, s, off, b, off, n, off % 4 == 0)
        state.rt.synth_q4(seed, i, SIGMA, 0, n, k, job)
        jobs.append(job)
    return jobs


def prepare(case, seed):
    state = State()
    state.kind = case["kind"]
    state.stream = torch.cuda.current_stream().cuda_stream
    if case["kind"] == "token":
        state.stack = SyntheticStack(state.rt, layers=case["layers"], vocab=case["vocab"], seed=seed)
        state.stack.reset_input(state.stream)
        state.chain = state.stack.build_chain()
        # the chain's first stage reads x and later stages write it: a token starts from the embedding
        state.embedding = state.stack.x.clone()
        return state
    state.m, state.k = case["m"], case["k"]
    state.dtype = capi.Q4B_F32 if case["dtype"] == "f32" else capi.Q4B_BF16
    state.jobs = _weights(state, case, seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    state.x = torch.randn(case["m"], case["k"], generator=gen, device="cuda")
    if case["kind"] in ("host", "host_mlp"):
        state.x = state.x.cpu().numpy().reshape(-1)
        return state
    if case["dtype"] == "bf16":
        state.x = state.x.to(torch.bfloat16)
    if case["kind"] == "argmax":
        state.tokens = torch.zeros(case["m"], dtype=torch.int32, device="cuda")
        state.values = torch.zeros(case["m"], dtype=torch.float32, device="cuda")
        return state
    rows = [case["k"]] if case["kind"] == "mlp" else [j.output_rows for j in state.jobs]
    state.outs = [torch.zeros(case["m"], n, device="cuda") for n in rows]
    state.flags = 0
    if case.get("residual"):
        state.flags = capi.FLAG_ACCUMULATE
        for o in state.outs:
            o.normal_(generator=gen)
    return state


def run(state):
    rt = state.rt
    if state.kind == "project":
        rt.matmul_batch_device(state.x.data_ptr(), state.dtype, state.m, state.k, state.jobs,
                               [o.data_ptr() for o in state.outs], state.flags, state.stream)
        return state.outs
    if state.kind == "mlp":
        rt.mlp_batch_device(state.x.data_ptr(), state.dtype, state.m, state.k, *state.jobs, state.outs[0].data_ptr(),
                            state.stream)
        return state.outs
    if state.kind == "argmax":
        rt.argmax_batch_device(state.x.data_ptr(), state.dtype, state.m, state.k, state.jobs[0], 0,
                               state.tokens.data_ptr(), state.values.data_ptr(), state.stream)
        return {"tokens": state.tokens, "values": state.values}
    if state.kind == "token":
        st = state.stack
        st.x.copy_(state.embedding)
        state.chain.run(state.stream)
        return {"token": st.token, "best": st.best, "logits": st.logits, "down": st.d, "hidden": st.h, "x": st.x,
                "projections": st.outs}
    if state.kind == "host":
        return rt.q4_affine_matmul_mapped_batch(state.x, state.m, state.jobs)
    return rt.q4_affine_mlp_mapped_batch(state.x, state.m, *state.jobs)


def work(case):
    """Packed weights, scales and biases (0.5625 bytes per weight) and the activation read once, results written once
    (read too in the residual form); a multiply and an add per weight and row."""
    shapes = _shapes(case)
    m = case.get("m", 1)
    weights = sum(n * k for n, k in shapes)
    size = 4 if case.get("dtype") == "f32" else 2
    if case["kind"] == "token":
        io = 2 * HIDDEN + 4 * case["vocab"]
    elif case["kind"] == "argmax":
        io = m * (size * case["k"] + 8)
    elif case["kind"] in ("mlp", "host_mlp"):
        io = m * case["k"] * (size + 4)
    else:
        io = m * (size * case["k"] + sum(n for n, _ in shapes) * (8 if case.get("residual") else 4))
    return {"bytes": weights * 9 // 16 + io, "flops": 2 * m * weights}


def tolerance(case):
    """Decode and short batches sum in 32 bits (1e-5). From 16 rows the tensor-core path rounds weights and
    activations to bf16 (2^-9 each, averaged over a dot product), and the MLP its hidden rows too. The chain rounds
    hidden and normalised vectors to bf16 between its stages."""
    if case["kind"] == "token":
        return {"rel": 4e-3, "max": 0.1}
    if case["m"] >= 16:
        return {"rel": 3e-3 if "mlp" not in case["kind"] else 5e-3}
    return {"rel": 1e-5 if "mlp" not in case["kind"] else 2e-5}
