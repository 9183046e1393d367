"""Prompt processing through the engine: several consecutive tokens of ONE sequence per step (chunks of up to 256
tokens, of max_batch where predictor logits are traced), K / V of the whole chunk stored first, causal attention after, union list for
reading and each token's own mask for writing.  Held against (1) the reference's llama.cpp logits after its own batched prompt (golden fixtures: the
reference's batched and token-by-token prompts give identical logits at one thread) and (2) the same engine fed the prompt
one token per step: the KV cache rows a chunk leaves behind must be what single steps leave."""
import os

import numpy as np
import pytest

import make_golden as mg
from powerinfer_b200 import synth
from test_gpu_engine import GOLD, tol

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def engine_mod():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from powerinfer_b200 import engine
    return engine


@pytest.mark.parametrize("name", ["llama_f16", "llama_q4_0", "llama_gqa_f16", "falcon_f16", "opt_f16"])
@pytest.mark.parametrize("max_batch", [8, 3])
def test_prompt_in_chunks_matches_the_reference_after_its_batched_prompt(engine_mod, name, max_batch):
    spec = mg.MODEL_CASES[name]
    g = np.load(os.path.join(GOLD, f"model_{name}.npz"))
    assert bool(g["single_equals_batch"])
    eng = engine_mod.DecodeEngine(spec, synth.build_model(spec), max_batch=max_batch)
    toks = [int(v) for v in g["prompt"]]                       # 8 tokens: one chunk, within a decode step's batch or larger than it
    logits, amax = eng.prefill(toks, seq=0, pos0=0)
    err = [float(np.abs(logits - g["logits"][0]).max())]
    assert amax == int(logits.argmax())
    cur, pos = int(g["greedy"][0]), len(toks)
    for s in range(1, 8):                                      # a few decode steps on top of the chunk-made KV cache
        lg, _ = eng.decode([cur], [pos])
        err.append(float(np.abs(lg[0] - g["logits"][s]).max()))
        cur, pos = int(g["greedy"][s]), pos + 1
    eng.status()
    eng.close()
    # a borderline neuron (predictor logit within rounding of the threshold) may flip between the batched and the reference's
    # kernels and move one step by that neuron's contribution: the bar must hold for nearly all steps, the median far inside
    assert np.mean(np.array(err) <= tol(spec)) >= 0.75 and np.median(err) <= 5e-3, err


@pytest.mark.parametrize("name", ["llama_q4_0", "falcon_f16"])
def test_chunked_prompt_leaves_the_kv_cache_single_steps_leave(engine_mod, name):
    spec = mg.MODEL_CASES[name]
    t = synth.build_model(spec)
    toks = [int(v) for v in np.random.default_rng(3).integers(3, spec.n_vocab, 21)]
    a = engine_mod.DecodeEngine(spec, t, max_batch=1)
    for p, tk in enumerate(toks):
        a.decode([tk], [p], want_logits=False)
    ref_l, _ = a.decode([5], [len(toks)])
    ka, va = a.k_cache.clone(), a.v_cache.clone()
    a.close()
    b = engine_mod.DecodeEngine(spec, t, max_batch=8)
    b.prefill(toks, seq=0, pos0=0, want_logits=False)           # one chunk of 21, no lm head at all
    got_l, _ = b.decode([5], [len(toks)])
    kb = b.k_cache.view(spec.n_layer, 8, spec.n_ctx, -1)[:, 0, :len(toks) + 1]
    vb = b.v_cache.view(spec.n_layer, 8, spec.n_ctx, -1)[:, 0, :len(toks) + 1]
    ka = ka.view(spec.n_layer, 1, spec.n_ctx, -1)[:, 0, :len(toks) + 1]
    va = va.view(spec.n_layer, 1, spec.n_ctx, -1)[:, 0, :len(toks) + 1]
    assert float((ka.float() - kb.float()).abs().max()) <= 2e-2 and float((va.float() - vb.float()).abs().max()) <= 2e-2
    assert np.abs(got_l[0] - ref_l[0]).max() <= tol(spec)
    b.status()
    b.close()


@pytest.mark.parametrize("n", [1, 21, 60])
def test_decoding_goes_on_from_the_device_after_a_prompt(engine_mod, n):
    """An engine for one sequence: after a prompt its I/O buffers hold the last token, its position and its greedy id, as after a step, so
    that pi_engine_advance feeds the next step without the host."""
    spec = mg.MODEL_CASES["llama_f16"]
    t = synth.build_model(spec)
    toks = [int(v) for v in np.random.default_rng(n).integers(3, spec.n_vocab, n)]
    eng = engine_mod.DecodeEngine(spec, t, max_batch=1)
    _, cur = eng.prefill(toks)
    want = []
    for pos in range(n, n + 4):
        cur = int(eng.decode([cur], [pos])[1][0])
        want.append(cur)
    eng.k_cache.zero_(); eng.v_cache.zero_(); torch.cuda.synchronize()
    eng.prefill(toks)
    got = []
    for pos in range(n, n + 4):
        eng.advance(1)
        eng.stream.synchronize()
        assert int(eng.device_view("pos", 1).cpu()[0]) == pos
        eng.step_device(1)
        eng.stream.synchronize()
        got.append(int(eng.device_view("argmax", 1).cpu()[0]))
    assert got == want
    eng.close()


def apart(spec, t, seed):
    """Second predictor matrices that keep every neuron's logit five standard deviations away from the threshold: kernels that add in another
    order choose the same neurons."""
    rng = np.random.default_rng(seed)
    for il in range(spec.n_layer):
        z = np.where(rng.random(spec.n_ff) < spec.firing, 5.0, -5.0)
        w = rng.standard_normal((spec.n_ff, spec.rank)) * spec.sigma
        t[f"blk.{il}.fc2.weight"] = (w + (spec.sigma / (0.564 * spec.rank ** 0.5) * z)[:, None]).astype(np.float16)
    return t


def against_single_steps(engine_mod, spec, lengths):
    t = apart(spec, synth.build_model(spec), 17)
    one, many = engine_mod.DecodeEngine(spec, t, max_batch=1), engine_mod.DecodeEngine(spec, t, max_batch=2)
    rng = np.random.default_rng(18)
    for n in lengths:
        toks = rng.integers(0, spec.n_vocab, n).astype(np.int32)
        for pos in range(n):
            ref, _ = one.decode([toks[pos]], [pos])
        got, got_id = many.prefill(toks, seq=1)
        # the bound of test_gpu_batches.test_prompt_chunks: roundings between the nodes that flip by one level
        assert np.linalg.norm(got - ref[0]) <= (24e-3 if spec.wtype == synth.Q4_0 else 3e-3) * np.linalg.norm(ref[0]), n
        assert got_id == int(got.argmax())
        a = one.k_cache.view(spec.n_layer, 1, spec.n_ctx, -1)[:, 0, :n].float()
        b = many.k_cache.view(spec.n_layer, 2, spec.n_ctx, -1)[:, 1, :n].float()
        assert (a - b).norm() <= (24e-3 if spec.wtype == synth.Q4_0 else 3e-3) * a.norm()
    many.status()
    one.close()
    many.close()


@pytest.mark.parametrize("wtype", [synth.F16, synth.Q4_0])
def test_prompt_over_many_neurons_per_cta(engine_mod, wtype):
    """277 neurons per CTA: the predictor's masks and the gather take several tiles of every token count."""
    against_single_steps(engine_mod, synth.ModelSpec(arch=synth.ARCH_LLAMA, wtype=wtype, n_layer=1, d=256, n_ff=40960, n_head=4, n_head_kv=4, rank=64, n_vocab=256,
                                                     n_ctx=256, firing=0.9, seed=6), (40, 77, 130, 256))


def test_prompt_with_rounded_factors(engine_mod):
    """Q4_0 prompts of an engine for several sequences at a width of whole 1024 columns: the down projection's factors are rounded to FP16, in
    token groups of 40, 48 and 64."""
    against_single_steps(engine_mod, synth.ModelSpec(arch=synth.ARCH_LLAMA, wtype=synth.Q4_0, n_layer=1, d=1024, n_ff=2048, n_head=8, n_head_kv=8, rank=64, n_vocab=256,
                                                     n_ctx=256, firing=0.5, seed=9), (40, 48, 90, 130))


@pytest.mark.parametrize("heads,kv,n_ctx", [(4, 4, 2048), (8, 2, 2304), (4, 2, 4096)])
def test_prompt_in_a_long_context(engine_mod, heads, kv, n_ctx):
    """Contexts beyond 1920 positions (heads of 64: 2112): chunks of 32 tokens and more with 24 CTAs and more (here 40 tokens of 8 heads, and 256) take the
    several-token attention up to 2880 (3136), all others and the longer contexts a store pass, then one CTA per head and token."""
    against_single_steps(engine_mod, synth.ModelSpec(arch=synth.ARCH_LLAMA, wtype=synth.F16, n_layer=2, d=512, n_ff=1024, n_head=heads, n_head_kv=kv, rank=64, n_vocab=256,
                                                     n_ctx=n_ctx, firing=0.2, seed=7), (2, 40, 300))


@pytest.mark.parametrize("heads,kv,n_ctx", [(4, 4, 2880), (4, 4, 2881), (8, 2, 3136), (8, 2, 3137)])
def test_prompt_in_a_context_at_the_line(engine_mod, heads, kv, n_ctx):
    test_prompt_in_a_long_context(engine_mod, heads, kv, n_ctx)


@pytest.mark.parametrize("wtype", [synth.F16, synth.Q4_0])
def test_prompt_in_a_workspace_with_room_for_fewer_partial_vectors(engine_mod, monkeypatch, wtype):
    """A workspace of the size that engines had before k_axpy_tc is taken, and their down projections are k_axpy_mm's: against the same prompts
    token by token."""
    from powerinfer_b200._lib import PiError
    spec = synth.ModelSpec(arch=synth.ARCH_LLAMA, wtype=wtype, n_layer=1, d=2048, n_ff=2048, n_head=16, n_head_kv=4, rank=64, n_vocab=256, n_ctx=256, firing=0.6, seed=9)
    t = apart(spec, synth.build_model(spec), 17)
    query = engine_mod.lib.pi_engine_workspace_bytes

    def engine_of(less):
        monkeypatch.setattr(engine_mod.lib, "pi_engine_workspace_bytes", lambda cfg: query(cfg) - less)
        try:
            return engine_mod.DecodeEngine(spec, t, max_batch=2)
        finally:
            monkeypatch.setattr(engine_mod.lib, "pi_engine_workspace_bytes", query)

    whole = engine_of(0)
    lo, hi = 0, query(engine_mod.C.byref(whole.cfg))                  # the most bytes that can be left out lie between
    whole.close()
    while hi - lo > 65536:
        mid = (lo + hi) // 2
        try:
            engine_of(mid).close()
            lo = mid
        except PiError:
            hi = mid
    assert lo > 1 << 20                                               # (some partial vectors of 256 tokens)
    small = engine_of(lo)
    one = engine_mod.DecodeEngine(spec, t, max_batch=1)
    rng = np.random.default_rng(18)
    for n in (50, 77, 200):
        toks = rng.integers(0, spec.n_vocab, n).astype(np.int32)
        for pos in range(n):
            ref, _ = one.decode([toks[pos]], [pos])
        got, _ = small.prefill(toks, seq=1)
        assert np.linalg.norm(got - ref[0]) <= (24e-3 if wtype == synth.Q4_0 else 3e-3) * np.linalg.norm(ref[0]), n
    small.status()
    one.close()
    small.close()


@pytest.mark.parametrize("wtype", [synth.F16, synth.Q4_0])
def test_prompt_in_chunks_of_the_batch(engine_mod, wtype):
    """With a trace of the predictor logits a prompt goes through in steps of max_batch tokens (8 + 8 + 5: a plain run, a captured one, a
    replay), and leaves what one chunk leaves."""
    spec = synth.ModelSpec(arch=synth.ARCH_LLAMA, wtype=wtype, n_layer=2, d=512, n_ff=1024, n_head=4, n_head_kv=2, rank=64, n_vocab=256, n_ctx=128, firing=0.2, seed=8)
    t = apart(spec, synth.build_model(spec), 8)
    toks = np.random.default_rng(8).integers(0, spec.n_vocab, 21)
    plain, traced = engine_mod.DecodeEngine(spec, t, max_batch=8), engine_mod.DecodeEngine(spec, t, max_batch=8)
    traced.enable_trace()
    want, want_id = plain.prefill(toks)
    for _ in range(3):
        got, got_id = traced.prefill(toks)
        assert np.linalg.norm(got - want) <= (24e-3 if wtype == synth.Q4_0 else 3e-3) * np.linalg.norm(want)
        assert got_id == int(got.argmax()) and want_id == int(want.argmax())
    plain.close()
    traced.close()
