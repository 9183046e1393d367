"""What is timed when this framework is timed: one pass of each case goes through the public entry points exactly as a
program that serves a model would call them.

Four kinds of case:

    decode    one step of `engine.DecodeEngine.decode`: a new token for each of `batch` sequences, token ids and positions
              from host memory, the logits back in host memory
    prefill   one prompt through `DecodeEngine.prefill`: consecutive tokens of one sequence in chunks of `batch`
    ffn       one call of `ggml_ops.sparse_ffn`: the whole neuron-sparse FFN of a layer for given predictor logits
    nodes     the same FFN node by node, as a graph over the ggml operators issues it: predictor, ggml_mul_mat_idx (up and
              gate), relu and product, ggml_axpy, over the share `held` of the neurons that this device holds (gpu_bucket)

The layers have the shapes of `powerinfer_b200.configs`.  An engine case holds fewer layers than the configuration (the
time of a step grows linearly with the layers); a layer's weights are still larger than L2, so no pass finds them there.

Weights are seeded random draws.  In the engine cases the second predictor matrix is drawn so that a neuron's logit lies
five standard deviations above the threshold or five below it, as training pushes a predictor's logits apart: two correct
implementations that add in another order then choose the same neurons.  The share of neurons above it is that of the
union, over the tokens of one step, of masks that fire with the mean `firing` on a Zipf(1.1) profile.  The operator cases
take masks of that profile themselves, another one for each token.
"""
import math

import numpy as np
import torch

from powerinfer_b200 import engine, ggml_ops, synth, synth_device
from powerinfer_b200._lib import check, lib

ARCHS = {"llama": synth.ARCH_LLAMA, "bamboo": synth.ARCH_LLAMA, "falcon": synth.ARCH_FALCON, "opt": synth.ARCH_OPT}
WTYPES = {"f16": synth.F16, "q4_0": synth.Q4_0}


def _engine(kind, arch, wtype, n_layer, d, n_ff, n_head, n_head_kv, rank, n_vocab, n_ctx, firing, batch, **more):
    return dict(kind=kind, arch=arch, wtype=wtype, n_layer=n_layer, d=d, n_ff=n_ff, n_head=n_head, n_head_kv=n_head_kv, rank=rank,
                n_vocab=n_vocab, n_ctx=n_ctx, firing=firing, batch=batch, **more)


def listed():
    llama7b = dict(arch="llama", wtype="f16", d=4096, n_ff=11008, n_head=32, n_head_kv=32, rank=1024, n_vocab=32000, n_ctx=512, firing=0.10)
    llama70b = dict(arch="llama", wtype="q4_0", d=8192, n_ff=28672, n_head=64, n_head_kv=8, rank=1024, n_vocab=32000, n_ctx=768, firing=0.12)
    return [
        # a model small enough that only launches and latency count (a draft model, a smoke test)
        dict(_engine("decode", "llama", "q4_0", 2, 512, 2048, 4, 2, 64, 512, 128, 0.15, 1, pos=40), name="decode small q4_0 x1"),
        # interactive generation with the 7B shape, in the middle of a reply
        dict(_engine("decode", n_layer=12, batch=1, pos=150, **llama7b), name="decode 7b f16 x1"),
        # interactive generation with the 70B shape: the headline of the benchmark
        dict(_engine("decode", n_layer=8, batch=1, pos=383, **llama70b), name="decode 70b q4_0 x1"),
        # interactive generation with the falcon graph: two norms of one input, one residual sum, 8 KV heads of 64
        dict(_engine("decode", "falcon", "f16", 4, 8192, 32768, 128, 8, 1024, 65024, 512, 0.10, 1, pos=255), name="decode 40b f16 x1"),
        # a handful of users served together: the predictors' union decides what is read
        dict(_engine("decode", n_layer=3, batch=8, pos=383, **llama70b), name="decode 70b q4_0 x8"),
        # the opt graph (biases, LayerNorm, relu(up + b)) with a small odd batch, layers of the largest shape
        dict(_engine("decode", "opt", "f16", 1, 12288, 49152, 96, 96, 1536, 50272, 512, 0.08, 5, pos=201), name="decode 175b opt f16 x5"),
        # the largest batch
        dict(_engine("decode", n_layer=8, batch=32, pos=190, **llama7b), name="decode 7b f16 x32"),
        # a prompt of the benchmark's length with the 70B shape
        dict(_engine("prefill", n_layer=3, batch=32, tokens=256, **llama70b), name="prefill 70b q4_0 256"),
        # a short prompt that is no multiple of the chunk
        dict(_engine("prefill", n_layer=8, batch=32, tokens=77, **llama7b), name="prefill 7b f16 77"),
        # one layer's FFN as a call of its own: a single token, 90 % sparse
        dict(kind="ffn", wtype="f16", d=5120, n_ff=13824, gated=True, firing=0.10, batch=1, name="ffn 13b f16 x1"),
        # a batch with less sparsity
        dict(kind="ffn", wtype="q4_0", d=5120, n_ff=13824, gated=True, firing=0.20, batch=16, name="ffn 13b q4_0 x16"),
        # the graph's nodes one by one over the hot half of the neurons (the hybrid split)
        dict(kind="nodes", wtype="q4_0", d=8192, n_ff=28672, rank=1024, firing=0.12, held=0.5, batch=1, name="nodes 70b q4_0 x1"),
    ]


def _log_uniform(rng, lo, hi, step):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step or step


def draw(rng):
    worst = max(_cost(c) for c in listed())
    while True:
        c = _draw(rng)
        if _cost(c) <= 0.6 * worst:
            return c


def _draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prefill", "ffn", "ffn", "nodes"])
    wtype = rng.choice(["f16", "q4_0"])
    batch = rng.choice([1, 1, _log_uniform(rng, 2, 32, 1)])
    firing = round(math.exp(rng.uniform(math.log(0.05), math.log(0.4))), 3)
    d = _log_uniform(rng, 512, 8192, 256)
    n_ff = int(d * rng.uniform(2.5, 4.0)) // 32 * 32
    if kind == "ffn":
        return dict(kind=kind, wtype=wtype, d=d, n_ff=n_ff, gated=rng.random() < 0.7, firing=firing, batch=batch)
    rank = _log_uniform(rng, 128, 1536, 8)
    if kind == "nodes":
        return dict(kind=kind, wtype=wtype, d=d, n_ff=n_ff, rank=rank, firing=firing, held=rng.choice([1.0, round(rng.uniform(0.2, 0.9), 2)]), batch=batch)
    arch = rng.choice(["llama", "llama", "bamboo", "falcon", "opt"])
    hd = rng.choice([64, 128])
    heads = d // hd
    kv = heads if arch == "opt" else heads // rng.choice([g for g in (1, 2, 4, 8, 16) if heads % g == 0])
    n_ctx = _log_uniform(rng, 128, 2048, 32)
    case = _engine(kind, arch, wtype, rng.randint(1, 8 if wtype == "f16" else 3), d, n_ff, heads, kv, rank, rng.randint(500, 65000), n_ctx, firing, batch)
    if kind == "decode":
        case["pos"] = rng.randint(n_ctx // 8, n_ctx - 2)
    else:
        case["batch"] = rng.choice([8, 16, 32])
        case["tokens"] = rng.randint(2, min(256, n_ctx - 1))
    return case


# ---------------------------------------------------------------------------------------------- sizes

def _row(case, cols):
    return cols // 32 * 18 if case["wtype"] == "q4_0" else cols * 2


def _union(case, tokens):
    """Expected share of neurons that fire for at least one of `tokens` tokens."""
    p = synth.zipf_profile(case["n_ff"], case["firing"])
    return float((1.0 - (1.0 - p) ** tokens).mean())


def _held(case):
    """32-neuron blocks of the neurons that this device holds (a bucket holds whole blocks)."""
    return max(1, int(case["n_ff"] // 32 * case["held"]))


def _step(case):
    """Tokens of the case's fullest step."""
    return min(case["batch"], case["tokens"]) if case["kind"] == "prefill" else case["batch"]


def _weights(case):
    """(bytes of all weights that a step reads, multiply-adds of one token), the lm head apart from the layers."""
    d, F, R = case["d"], case["n_ff"], case["rank"]
    d_kv = d // case["n_head"] * case["n_head_kv"]
    mats = 3 if case["arch"] in ("llama", "bamboo") else 2
    live, own = _union(case, _step(case)) * F, case["firing"] * F
    attn, pred = d * (2 * d + 2 * d_kv), R * (d + F)
    layer = attn // d * _row(case, d) + 2 * pred + mats * live * _row(case, d)
    macs = attn + pred + mats * own * d
    head = case["n_vocab"] * (2 * d if case["arch"] == "opt" else _row(case, d))
    return case["n_layer"] * layer, head, case["n_layer"] * macs, case["n_vocab"] * d


def _cost(case):
    if case["kind"] in ("ffn", "nodes"):
        return work(case)["bytes"]
    layers, head, _, _ = _weights(case)
    return head + layers * (-(-case["tokens"] // case["batch"]) * case["batch"] / 8.0 if case["kind"] == "prefill" else max(1.0, case["batch"] / 8.0))


def work(case):
    T, d, F = case["batch"], case["d"], case["n_ff"]
    if case["kind"] in ("decode", "prefill"):
        layers, head, macs, head_macs = _weights(case)
        kv_row = 2 * case["n_layer"] * d // case["n_head"] * case["n_head_kv"] * 2                    # K and V of one position, all layers
        if case["kind"] == "decode":
            n, logits, seen, pairs = T, T, sum(_positions(case)) + T, sum(_positions(case)) + T
        else:
            n, logits, seen = case["tokens"], 1, case["tokens"]
            pairs = n * (n + 1) // 2
        return {"bytes": layers + head + kv_row * (seen + n) + 2 * n * d + 4 * logits * case["n_vocab"],
                "flops": 2.0 * (macs * n + head_macs * logits + 2 * pairs * d * case["n_layer"])}
    live, own = _union(case, T) * F, case["firing"] * F
    if case["kind"] == "ffn":
        mats = 3 if case["gated"] else 2
        return {"bytes": mats * live * _row(case, d) + 4 * T * (F + 2 * d), "flops": 2.0 * mats * own * d * T}
    share = _held(case) * 32 / F
    return {"bytes": 2 * case["rank"] * (d + F) + 3 * share * live * _row(case, d) + 4 * T * (2 * d + 3 * F),
            "flops": 2.0 * T * (case["rank"] * (d + F) + 3 * share * own * d)}


def tolerance(case):
    if case["kind"] in ("decode", "prefill"):
        # Activations are rounded between the nodes, to FP16 (F16 weights) or to the int8 of Q8_0 (Q4_0 weights).  Sums in
        # another order flip some of these roundings, each by one level (2^-11, or 1/127 of a block's largest value), every
        # layer adds its own, and in a prompt every position reads the others'.  This framework's own kernels differ from
        # each other by up to 1.6e-3 (F16) and 2.2e-2 (Q4_0) at the listed cases.
        return {"rel": 3e-2, "max": 0.2} if case["wtype"] == "q4_0" else {"rel": 3e-3, "max": 0.03}
    # one layer's operators: FP32 sums, but the FFN rounds its hidden values on the way, to int8 in blocks of 32 (Q4_0) or to
    # FP16, and a batch of Q4_0 may round weight and coefficient of the down projection to FP16 once each
    return {"rel": 2e-3, "max": 0.02} if case["wtype"] == "q4_0" else {"rel": 2e-4, "max": 2e-3}


# ---------------------------------------------------------------------------------------------- preparation

def _spec(case):
    return synth.ModelSpec(arch=ARCHS[case["arch"]], wtype=WTYPES[case["wtype"]], n_layer=case["n_layer"], d=case["d"], n_ff=case["n_ff"],
                           n_head=case["n_head"], n_head_kv=case["n_head_kv"], rank=case["rank"], n_vocab=case["n_vocab"], n_ctx=case["n_ctx"],
                           firing=case["firing"], gate_sym=case["arch"] == "bamboo")


def _fc2(gen, rows, rank, live, sigma=0.02):
    """Second predictor matrix: `live` of the rows (a random choice) lie five standard deviations above the threshold, the
    others as far below (the mean of a row makes the logit's mean, see powerinfer_b200.synth)."""
    z = torch.full((rows,), -5.0, device="cuda")
    z[torch.randperm(rows, device="cuda", generator=gen)[:max(1, round(live * rows))]] = 5.0
    w = torch.randn(rows, rank, device="cuda", generator=gen) * sigma
    return (w + (sigma / (0.564 * math.sqrt(rank)) * z)[:, None]).to(torch.float16)


def _positions(case):
    """Sequences of a batch are at different positions."""
    return [max(0, case["pos"] - 5 * t) for t in range(case["batch"])]


def _prepare_engine(case, seed):
    spec = _spec(case)
    tensors, layers = synth_device.build_local_model(spec, seed=seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    live = _union(case, _step(case))
    for layer in layers:
        layer["fc2"] = _fc2(gen, spec.n_ff, spec.rank, live)
    eng = engine.DecodeEngine(spec, tensors, max_batch=case["batch"], local_layers=layers)
    n = case["tokens"] if case["kind"] == "prefill" else case["batch"]
    tokens = np.random.default_rng(seed).integers(0, spec.n_vocab, n).astype(np.int32)
    eng.k_cache.normal_(generator=gen)                 # earlier positions, and the sequences of other users, hold keys and
    eng.v_cache.normal_(generator=gen)                 # values already
    torch.cuda.synchronize()                           # the engine runs on a stream of its own
    return dict(kind=case["kind"], eng=eng, tokens=tokens, pos=np.array(_positions(case), np.int32) if case["kind"] == "decode" else None)


def _weight(gen, wtype, rows, cols, keep=None):
    w = (torch.randn(rows, cols, device="cuda", generator=gen) * 0.02).to(torch.float16)
    if keep is not None:
        w = w[keep].contiguous()
        rows = w.shape[0]
    if wtype == synth.F16:
        return ggml_ops.Weight(wtype, w.view(torch.uint8).reshape(-1), rows, cols)
    raw = ggml_ops.quantize_q4_0(w.float())
    planar = torch.empty_like(raw)
    check(lib.pi_q4_0_repack(raw.data_ptr(), planar.data_ptr(), rows, cols, torch.cuda.current_stream().cuda_stream))
    return ggml_ops.Weight(wtype, planar, rows, cols)


def _prepare_op(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    wtype, d, F, T = WTYPES[case["wtype"]], case["d"], case["n_ff"], case["batch"]
    x = torch.randn(T, d, device="cuda", generator=gen)
    if case["kind"] == "ffn":
        profile = torch.from_numpy(synth.zipf_profile(F, case["firing"])).float().cuda()[torch.randperm(F, device="cuda", generator=gen)]
        logits = torch.rand(T, F, device="cuda", generator=gen)
        idx = torch.where(logits < profile[None, :], logits + 0.01, -logits - 0.01)
        up = _weight(gen, wtype, F, d)
        gate = _weight(gen, wtype, F, d) if case["gated"] else None
        bias = None if case["gated"] else torch.randn(F, device="cuda", generator=gen) * 0.1
        return dict(kind="ffn", up=up, gate=gate, down=_weight(gen, wtype, F, d), x=x, idx=idx, bias=bias)
    bucket = keep = None
    if case["held"] < 1.0:                             # whole blocks of 32 neurons, in order
        blocks = torch.sort(torch.randperm(F // 32, device="cuda", generator=gen)[:_held(case)])[0]
        keep = (blocks[:, None] * 32 + torch.arange(32, device="cuda")[None, :]).reshape(-1)
        bucket = keep.to(torch.int32)
    fc1 = _weight(gen, synth.F16, case["rank"], d)
    fc2 = _fc2(gen, F, case["rank"], _union(case, T))
    return dict(kind="nodes", fc1=fc1, fc2=ggml_ops.Weight(synth.F16, fc2.view(torch.uint8).reshape(-1), F, case["rank"]), x=x, F=F, bucket=bucket,
                up=_weight(gen, wtype, F, d, keep), gate=_weight(gen, wtype, F, d, keep), down=_weight(gen, wtype, F, d, keep))


def prepare(case, seed):
    state = _prepare_engine(case, seed) if case["kind"] in ("decode", "prefill") else _prepare_op(case, seed)
    torch.cuda.synchronize()
    return state


# ---------------------------------------------------------------------------------------------- the pass

def run(state):
    if state["kind"] == "decode":
        # (the greedy ids come back too; they follow from the logits and are no output of their own: a near tie may go
        # either way under the logits' tolerance)
        logits, _ = state["eng"].decode(state["tokens"], state["pos"])
        return {"logits": logits, "k_cache": state["eng"].k_cache, "v_cache": state["eng"].v_cache}
    if state["kind"] == "prefill":
        logits, _ = state["eng"].prefill(state["tokens"])
        return {"logits": logits, "k_cache": state["eng"].k_cache, "v_cache": state["eng"].v_cache}
    if state["kind"] == "ffn":
        return ggml_ops.sparse_ffn(state["up"], state["gate"], state["down"], state["x"], state["idx"], up_bias=state["bias"])
    idx = ggml_ops.predictor(state["fc1"], state["fc2"], state["x"])
    up = ggml_ops.ggml_mul_mat_idx(state["up"], state["x"], idx, state["bucket"], state["F"])
    gate = ggml_ops.ggml_mul_mat_idx(state["gate"], state["x"], idx, state["bucket"], state["F"])
    h = torch.relu(gate) * up
    return idx, h, ggml_ops.ggml_axpy(state["down"], h, idx, state["bucket"])
