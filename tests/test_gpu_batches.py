"""Kernels of steps with several tokens at the sizes where their work split can go wrong: rows and columns that are no multiple of a
tile, one row per CTA and several tiles per CTA, token counts around every boundary of the dispatch (8, 16, 24, 32, 64, 128, 256).

The reference is the same sum in float64 over the values that the kernel multiplies: FP16-rounded activations with F16 weights, the
dequantised Q8_0 activation with dequantised Q4_0 weights.  What is left between the two is FP32 accumulation: at most one rounding of
2^-24 per term (three more per block of 32 for the Q4_0 scales), so |error| <= (n + 8) 2^-24 sum |w x|.
"""
import numpy as np
import pytest

from powerinfer_b200 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TOKENS = [2, 8, 9, 16, 17, 24, 25, 32, 33, 48, 64, 65, 77, 96, 128, 129, 256, 261]


def weight(ops, wtype, rows, cols, gen):
    w = torch.randn(rows, cols, device="cuda", generator=gen) * 0.05
    if wtype == synth.F16:
        return ops.upload_weight(w.half().cpu().numpy(), wtype, rows, cols)
    return ops.upload_weight(synth.quantize_q4_0(w.cpu().numpy()), wtype, rows, cols)


def rounded(ops, wtype, x):
    """the activation as the weights of this type consume it, float64"""
    if wtype == synth.F16:
        return x.half().double()
    q = ops.quantize_q8_0(x).cpu().numpy().reshape(-1, 34)
    d = q[:, :2].copy().view(np.float16).astype(np.float64)
    return torch.from_numpy((d * q[:, 2:].view(np.int8)).reshape(x.shape)).cuda()


def close(got, x, w, keep=None):
    ref, mass = x @ w.T, x.abs() @ w.abs().T
    if keep is not None:
        ref, mass = ref * keep, mass * keep
    bound = (x.shape[1] + 8) * 2.0 ** -24 * mass + 1e-30
    worst = ((got.double() - ref).abs() / bound).max().item()
    assert worst <= 1.0, worst


@pytest.mark.parametrize("wtype,rows,cols", [(synth.F16, 33, 72), (synth.F16, 5000, 264), (synth.F16, 40960, 136), (synth.F16, 1031, 4104),
                                             (synth.Q4_0, 40, 256), (synth.Q4_0, 5001, 512), (synth.Q4_0, 40959, 256), (synth.Q4_0, 1031, 4352)])
def test_dense_and_gather(wtype, rows, cols):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from powerinfer_b200 import ggml_ops as ops
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rows)
    W = weight(ops, wtype, rows, cols, gen)
    w = ops.dequantize(W).double()
    bucket = torch.sort(torch.randperm(rows + 37, device="cuda", generator=gen)[:rows])[0].to(torch.int32)
    for T in TOKENS:
        x = torch.randn(T, cols, device="cuda", generator=gen)
        bias = torch.randn(rows, device="cuda", generator=gen)
        xr = rounded(ops, wtype, x)
        close(ops.ggml_mul_mat(W, x), xr, w)
        got = ops.ggml_mul_mat(W, x, bias)
        assert torch.allclose(got.double(), xr @ w.T + bias, rtol=1e-5, atol=1e-4)
        for idx in (torch.randn(T, rows, device="cuda", generator=gen) - 1.0, torch.full((T, rows), -1.0, device="cuda")):   # some rows, none
            close(ops.ggml_mul_mat_idx(W, x, idx), xr, w, (idx >= 0).double())
        idx = torch.randn(T, rows + 37, device="cuda", generator=gen)
        got = ops.ggml_mul_mat_idx(W, x, idx, bucket, rows + 37)
        close(got[:, bucket.long()], xr, w, (idx[:, bucket.long()] >= 0).double())
        other = torch.ones(rows + 37, dtype=torch.bool, device="cuda")
        other[bucket.long()] = False
        assert not got[:, other].any()


@pytest.mark.parametrize("wtype,rows,cols", [(synth.F16, 2048, 264), (synth.F16, 4100, 1032), (synth.Q4_0, 2048, 256), (synth.Q4_0, 4128, 1024), (synth.Q4_0, 12320, 512)])
def test_axpy(wtype, rows, cols):
    """The coefficient is FP16(h), or the Q8_0 value of h in its block of 32 neurons (inactive ones included, as they stand in h); at widths
    of whole 1024 columns the Q4_0 kernel rounds weight and coefficient to FP16 once each: 2^-10 of a term."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from powerinfer_b200 import ggml_ops as ops
    gen = torch.Generator(device="cuda")
    gen.manual_seed(cols)
    W = weight(ops, wtype, rows, cols, gen)
    w = ops.dequantize(W).double()
    for T in TOKENS:
        for shift in (1.0, 100.0):                                    # some rows; none
            idx = torch.randn(T, rows, device="cuda", generator=gen) - shift
            h = torch.relu(torch.randn(T, rows, device="cuda", generator=gen)) * (idx >= 0)
            c = rounded(ops, wtype, h) * (idx >= 0)
            got = ops.ggml_axpy(W, h, idx).double()
            mass = c.abs() @ w.abs()
            per_term = (rows + 8) * 2.0 ** -24 + (2.0 ** -10 if wtype == synth.Q4_0 and cols % 1024 == 0 else 0.0)
            assert ((got - c @ w).abs() <= per_term * mass + 1e-30).all(), T


@pytest.mark.parametrize("heads,kv,hd", [(8, 2, 128), (9, 9, 128), (20, 20, 128), (34, 2, 128), (40, 40, 64)])
def test_attention_of_a_batch(heads, kv, hd):
    """Up to 32 sequences at different positions, CTAs for one and for several per SM.  With x = maximum - score, the kernel rounds x, exp(-x)
    and the probability to FP16 (2^-11 x, 2^-11, 2^-11 and 2^-25 for subnormals), and the normaliser carries the same errors averaged:
    |error| <= sum p (x + mean x + 5) 2^-11 |v| + 2^-24 sum |v|, the 5 with one unit for what FP32 sums and second-order terms add."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from powerinfer_b200 import ggml_ops as ops
    gen = torch.Generator(device="cuda")
    gen.manual_seed(heads)
    n_ctx, S = 160, 32
    for T in (2, 8, 32):
        kc = torch.randn(S, n_ctx, kv * hd, device="cuda", generator=gen).half()
        vc = torch.randn(S, n_ctx, kv * hd, device="cuda", generator=gen).half()
        q = torch.randn(T, heads * hd, device="cuda", generator=gen)
        k, v = (torch.randn(T, kv * hd, device="cuda", generator=gen) for _ in range(2))
        seq = torch.randperm(S, device="cuda", generator=gen)[:T].int()
        pos = torch.tensor([(0, 7, 63, 64, 130, 159)[t % 6] for t in range(T)], dtype=torch.int32, device="cuda")
        got = ops.attention_decode(q, k, v, kc, vc, pos, heads, kv, seq=seq).double().view(T, heads, hd)
        for t in range(T):
            s, n = int(seq[t]), int(pos[t]) + 1
            assert torch.equal(kc[s, n - 1], k[t].half()) and torch.equal(vc[s, n - 1], v[t].half())
            K, V = (c[s, :n].double().view(n, kv, hd).repeat_interleave(heads // kv, 1) for c in (kc, vc))
            sc = torch.einsum("hd,nhd->hn", q[t].half().double().view(heads, hd), K) / hd ** 0.5
            p, x = sc.softmax(1), sc.max(1, keepdim=True)[0] - sc
            w = p * (x + (p * x).sum(1, keepdim=True) + 5) * 2.0 ** -11 + 2.0 ** -24
            assert ((got[t] - torch.einsum("hn,nhd->hd", p, V)).abs() <= torch.einsum("hn,nhd->hd", w, V.abs())).all(), (T, t)


@pytest.mark.parametrize("arch,wtype,heads,kv,d", [(synth.ARCH_LLAMA, synth.F16, 8, 2, 512), (synth.ARCH_LLAMA, synth.Q4_0, 4, 4, 512), (synth.ARCH_OPT, synth.F16, 4, 4, 512),
                                                   (synth.ARCH_FALCON, synth.Q4_0, 32, 1, 2048), (synth.ARCH_LLAMA, synth.F16, 16, 16, 512)])
def test_prompt_chunks(arch, wtype, heads, kv, d):
    """A prompt in one chunk against the same prompt token by token (one-token kernels).  The second predictor matrix keeps every neuron's
    logit five standard deviations away from the threshold, so that both choose the same neurons (a neuron at the threshold that flips
    moves the logits by its whole contribution, whatever the kernels' precision).  Then the two differ by roundings of the activations
    between the nodes that flip by one level: 2^-11 for FP16 and 2^-8 of a block's maximum for Q8_0, about ten rounded vectors per layer
    that add like independent errors, in two layers: 4.5 x 2^-11 x sqrt(1 + 1/3) < 3e-3 of the norm, eight times that for Q8_0."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from powerinfer_b200 import engine
    spec = synth.ModelSpec(arch=arch, wtype=wtype, n_layer=2, d=d, n_ff=2048, n_head=heads, n_head_kv=kv, rank=64, n_vocab=515, n_ctx=320, firing=0.2, seed=heads)
    t = synth.build_model(spec)
    rng = np.random.default_rng(3)
    for il in range(spec.n_layer):
        z = np.where(rng.random(spec.n_ff) < spec.firing, 5.0, -5.0)
        w = rng.standard_normal((spec.n_ff, spec.rank)) * spec.sigma
        t[f"blk.{il}.fc2.weight"] = (w + (spec.sigma / (0.564 * spec.rank ** 0.5) * z)[:, None]).astype(np.float16)
    one, many = engine.DecodeEngine(spec, t, max_batch=1), engine.DecodeEngine(spec, t, max_batch=3)
    for n in (2, 33, 77, 256, 300):
        toks = rng.integers(0, spec.n_vocab, n).astype(np.int32)
        for pos in range(n):
            ref, ref_id = one.decode([toks[pos]], [pos])
        got, got_id = many.prefill(toks, seq=2)
        assert np.linalg.norm(got - ref[0]) <= (24e-3 if wtype == synth.Q4_0 else 3e-3) * np.linalg.norm(ref[0]), n
        assert got_id == int(got.argmax())
        assert ref_id[0] == int(ref[0].argmax())
    one.close()
    many.close()
