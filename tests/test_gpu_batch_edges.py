"""Steps with several tokens where a kernel's promise ends or its input is out of the ordinary: which Q4_0 down projections keep the CPU
path's 32-bit factors, rows of any bucket, values that are not finite, addresses that are aligned to one value only.

References are float64 sums over the values that the kernels multiply (Q8_0 activations with dequantised Q4_0 weights, FP16 with FP16).
"""
import numpy as np
import pytest

from powerinfer_b200 import synth
from test_gpu_batches import rounded, weight

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from powerinfer_b200 import ggml_ops
    return ggml_ops


def generator(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return gen


def few(gen, T, rows, n):
    """predictor logits under which the same `n` rows are active for every token"""
    idx = torch.full((T, rows), -1.0, device="cuda")
    on = torch.randperm(rows, device="cuda", generator=gen)[:n]
    idx[:, on] = 1.0
    return idx, on


@pytest.mark.parametrize("rows,T", [(64, 33), (64, 40), (96, 128), (64, 261), (262208, 2), (262208, 32)])
def test_axpy_keeps_32_bit_factors(ops, rows, T):
    """More than 32 tokens, or more than 2^28 weights, at a width where a smaller step rounds its factors to FP16.  Products of FP32 factors
    summed in FP32 are off by at most one rounding of 2^-24 per term and a few for each factor; FP16 factors would be off by 2^-11."""
    cols, n = 1024, 12
    gen = generator(rows + T)
    if rows > 10000:
        raw = ops.quantize_q4_0(torch.randn(rows, cols, device="cuda", generator=gen) * 0.05)
        planar = torch.empty_like(raw)
        from powerinfer_b200._lib import check, lib
        check(lib.pi_q4_0_repack(raw.data_ptr(), planar.data_ptr(), rows, cols, torch.cuda.current_stream().cuda_stream))
        W = ops.Weight(synth.Q4_0, planar, rows, cols)
    else:
        W = weight(ops, synth.Q4_0, rows, cols, gen)
    idx, on = few(gen, T, rows, n)
    h = torch.zeros(T, rows, device="cuda")
    h[:, on] = torch.rand(T, n, device="cuda", generator=gen) + 0.1
    w = ops.dequantize(W)[on].double()
    c = rounded(ops, synth.Q4_0, h)[:, on]
    got = ops.ggml_axpy(W, h, idx).double()
    assert ((got - c @ w).abs() <= (n + 8) * 2.0 ** -24 * (c.abs() @ w.abs())).all()


@pytest.mark.parametrize("n", [20, 40])
def test_prompt_of_an_engine_for_one_sequence_keeps_32_bit_factors(ops, n):
    """A prompt against the same prompt token by token, in a model where nothing but the FFN's sum can differ: one layer, no attention
    output, predictor logits far from the threshold.  Up to the axpy both make the same bits but for rare flips of an FP16 rounding in the
    norms' outputs.  Two sums of 32-bit products that add in another order are 1e-6 apart; FP16 factors (2^-11 / sqrt(3) for two random
    roundings of up to half a unit each) 2e-4."""
    from powerinfer_b200 import engine
    spec = synth.ModelSpec(arch=synth.ARCH_OPT, wtype=synth.Q4_0, n_layer=1, d=1024, n_ff=1024, n_head=8, n_head_kv=8, rank=64, n_vocab=512, n_ctx=64, firing=0.2, seed=5)
    t = synth.build_model(spec)
    rng = np.random.default_rng(5)
    z = np.where(rng.random(spec.n_ff) < spec.firing, 5.0, -5.0)
    w = rng.standard_normal((spec.n_ff, spec.rank)) * spec.sigma
    t["blk.0.fc2.weight"] = (w + (spec.sigma / (0.564 * spec.rank ** 0.5) * z)[:, None]).astype(np.float16)
    t["blk.0.attn_output.weight"] = np.zeros_like(t["blk.0.attn_output.weight"])
    one, many = engine.DecodeEngine(spec, t, max_batch=1), engine.DecodeEngine(spec, t, max_batch=1)
    toks = rng.integers(0, spec.n_vocab, n).astype(np.int32)
    for pos in range(n):
        ref, _ = one.decode([toks[pos]], [pos])
    got, _ = many.prefill(toks)
    one.close()
    many.close()
    assert np.linalg.norm(got - ref[0]) <= 4e-5 * np.linalg.norm(ref[0])


def axpy_close(got, c, w, cols, T):
    per_term = (w.shape[0] + 8) * 2.0 ** -24 + (2.0 ** -10 if cols % 1024 == 0 and T <= 32 else 0.0)
    assert ((got.double() - c @ w).abs() <= per_term * (c.abs() @ w.abs()) + 1e-30).all()


@pytest.mark.parametrize("cols", [256, 1024])
@pytest.mark.parametrize("T", [2, 9, 40])
def test_q8_blocks_are_those_of_the_global_neurons(ops, cols, T):
    """The coefficient's scale is that of the 32 neurons around it in h, whichever of them this device holds: any sorted bucket, a bucket of
    whole blocks that ends inside one, and rows that end inside a block of h."""
    gen = generator(cols + T)
    F = 640
    h = torch.randn(T, F, device="cuda", generator=gen) * torch.rand(1, F, device="cuda", generator=gen) ** 4
    idx = torch.randn(T, F, device="cuda", generator=gen)
    some = torch.sort(torch.randperm(F, device="cuda", generator=gen)[:333])[0]
    blocks = torch.cat([torch.arange(b * 32, b * 32 + 32, device="cuda") for b in (0, 3, 4, 9, 17)])[:-11]
    for ids in (some, blocks, torch.arange(600, device="cuda")):
        W = weight(ops, synth.Q4_0, len(ids), cols, gen)
        c = (rounded(ops, synth.Q4_0, h) * (idx >= 0))[:, ids]
        got = ops.ggml_axpy(W, h, idx, None if len(ids) == 600 else ids.int())
        axpy_close(got, c, ops.dequantize(W).double(), cols, T)


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("T", [2, 9, 40])
def test_sparse_ffn_of_any_bucket(ops, gated, T):
    """The whole FFN over any part of the neurons: neurons held elsewhere count as 0 in their blocks, held ones that are inactive as 0 or as
    relu(bias), as the graph's nodes leave them."""
    gen = generator(T)
    F, d = 640, 256
    ids = torch.sort(torch.randperm(F, device="cuda", generator=gen)[:333])[0]
    up, gate, down = (weight(ops, synth.Q4_0, len(ids), d, gen) for _ in range(3))
    x = torch.randn(T, d, device="cuda", generator=gen)
    idx = torch.randn(T, F, device="cuda", generator=gen)
    bias = None if gated else torch.randn(F, device="cuda", generator=gen)
    got = ops.sparse_ffn(up, gate if gated else None, down, x, idx, gpu_bucket=ids.int(), up_bias=bias)
    h = ops.ggml_mul_mat_idx(up, x, idx, ids.int(), F)
    if gated:
        h = torch.relu(ops.ggml_mul_mat_idx(gate, x, idx, ids.int(), F)) * h
    else:
        h[:, ids] = torch.relu(h[:, ids] + bias[ids])
    c = (rounded(ops, synth.Q4_0, h) * (idx >= 0))[:, ids]
    axpy_close(got, c, ops.dequantize(down).double(), d, T)


def attention_reference(q, k, v, heads, kv):
    """softmax(q k^T / sqrt(hd)) v of one token's heads in float64; k, v [n, kv * hd]"""
    n, hd = k.shape[0], q.numel() // heads
    K, V = (c.double().view(n, kv, hd).repeat_interleave(heads // kv, 1) for c in (k, v))
    sc = torch.einsum("hd,nhd->hn", q.half().double().view(heads, hd), K) / hd ** 0.5
    p, x = sc.softmax(1), sc.max(1, keepdim=True)[0] - sc
    w = p * (x + (p * x).sum(1, keepdim=True) + 5) * 2.0 ** -11 + 2.0 ** -24      # the bound of test_gpu_batches.test_attention_of_a_batch
    return torch.einsum("hn,nhd->hd", p, V), torch.einsum("hn,nhd->hd", w, V.abs())


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("T", [1, 3, 40])
def test_attention_result_at_any_float_address(ops, hd, T):
    """The F32 result goes to any address that is aligned to a float."""
    from powerinfer_b200._lib import check, lib
    gen = generator(hd + T)
    heads, kv, n_ctx = 4, 2, 64
    kc, vc = (torch.randn(T, n_ctx, kv * hd, device="cuda", generator=gen).half() for _ in range(2))
    q = torch.randn(T, heads * hd, device="cuda", generator=gen)
    k, v = (torch.randn(T, kv * hd, device="cuda", generator=gen) for _ in range(2))
    pos = torch.tensor([(40, 3, 63)[t % 3] for t in range(T)], dtype=torch.int32, device="cuda")
    seq = torch.arange(T, dtype=torch.int32, device="cuda")
    buf = torch.zeros(T * heads * hd + 8, device="cuda")
    for off in (0, 1, 2, 3):
        out = buf[off:off + T * heads * hd]
        buf.zero_()
        check(lib.pi_attention_decode(q.data_ptr(), k.data_ptr(), v.data_ptr(), kc.data_ptr(), vc.data_ptr(), seq.data_ptr(), pos.data_ptr(), T, heads, kv, hd, n_ctx,
                                      out.data_ptr(), torch.cuda.current_stream().cuda_stream))
        for t in range(T):
            ref, bound = attention_reference(q[t], kc[t, :int(pos[t]) + 1], vc[t, :int(pos[t]) + 1], heads, kv)
            assert ((out.double().view(T, heads, hd)[t] - ref).abs() <= bound).all(), (off, t)
        assert not buf[:off].any() and not buf[off + T * heads * hd:].any()


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("n", [20, 40])
def test_a_value_that_overflows_stays_with_the_tokens_that_see_it(ops, hd, n):
    """A prompt whose tenth token has values beyond FP16's range: the rows that the tokens before it leave in the next layer's cache are those
    of the same prompt without it.  (Its column of the value matrix is 0 times 60000 for every other token.)"""
    from powerinfer_b200 import engine
    spec = synth.ModelSpec(arch=synth.ARCH_LLAMA, wtype=synth.F16, n_layer=2, d=512, n_ff=1024, n_head=512 // hd, n_head_kv=512 // hd, rank=64, n_vocab=64, n_ctx=64, firing=0.2, seed=9)
    t = synth.build_model(spec)
    rng = np.random.default_rng(9)
    for il in range(spec.n_layer):
        z = np.where(rng.random(spec.n_ff) < spec.firing, 5.0, -5.0)
        w = rng.standard_normal((spec.n_ff, spec.rank)) * spec.sigma
        t[f"blk.{il}.fc2.weight"] = (w + (spec.sigma / (0.564 * spec.rank ** 0.5) * z)[:, None]).astype(np.float16)
    t["token_embd.weight"][:, 7] = 0
    t["token_embd.weight"][63] = 0
    t["token_embd.weight"][63, 7] = 1
    t["blk.0.attn_v.weight"][:, 7] = 60000
    toks = rng.integers(0, 63, n).astype(np.int32)
    toks[9] = 63
    rows = []
    for prompt in (toks, toks[:9]):
        eng = engine.DecodeEngine(spec, t, max_batch=1)
        eng.prefill(prompt, want_logits=False)
        torch.cuda.synchronize()
        rows.append(eng.k_cache.view(2, spec.n_ctx, -1)[1, :9].float().clone())
        assert torch.isinf(eng.v_cache.view(2, spec.n_ctx, -1)[0, 9]).all() == (len(prompt) > 9)
        eng.close()
    assert torch.isfinite(rows[0]).all()
    # FP16 roundings between the nodes that flip by one level, as in test_gpu_batches.test_prompt_chunks
    assert (rows[0] - rows[1]).norm() <= 3e-3 * rows[1].norm()


def test_dense_matrix_of_more_rows_than_a_tile_grid_takes(ops):
    """More than 2^26 rows and several tokens."""
    rows, cols, T = 2 ** 26 + 9, 8, 2
    gen = generator(1)
    w = torch.randint(-3, 4, (rows, cols), device="cuda", generator=gen, dtype=torch.int8).half()
    x = torch.randint(-3, 4, (T, cols), device="cuda", generator=gen, dtype=torch.int8).float()
    got = ops.ggml_mul_mat(ops.Weight(synth.F16, w.view(torch.uint8).reshape(-1), rows, cols), x)      # (small whole numbers: exact)
    assert torch.equal(got, x @ w.float().T)


@pytest.mark.parametrize("wtype,gated", [(synth.F16, True), (synth.F16, False), (synth.Q4_0, True)])
def test_gathers_of_more_rows_than_their_masks_are_scanned_for(ops, wtype, gated):
    """More than 262144 rows and several tokens: rows from a list, for up to 8 tokens at a time."""
    rows, cols = 262240, 64 if wtype == synth.F16 else 256
    gen = generator(rows)
    def w(rows, cols):
        if wtype == synth.F16:
            return ops.Weight(wtype, (torch.randn(rows, cols, device="cuda", generator=gen) * 0.05).half().view(torch.uint8).reshape(-1), rows, cols)
        raw = ops.quantize_q4_0(torch.randn(rows, cols, device="cuda", generator=gen) * 0.05)
        planar = torch.empty_like(raw)
        from powerinfer_b200._lib import check, lib
        check(lib.pi_q4_0_repack(raw.data_ptr(), planar.data_ptr(), rows, cols, torch.cuda.current_stream().cuda_stream))
        return ops.Weight(wtype, planar, rows, cols)
    up, gate, down = w(rows, cols), w(rows, cols), w(rows, cols)
    U, G, D = (ops.dequantize(m).double() for m in (up, gate, down))
    for T in (3, 13):
        x = torch.randn(T, cols, device="cuda", generator=gen)
        idx, on = few(gen, T, rows, 3000)
        idx[:, on] -= torch.rand(T, len(on), device="cuda", generator=gen) * 1.5                   # active for some tokens
        xr, keep = rounded(ops, wtype, x), (idx[:, on] >= 0).double()
        got = ops.ggml_mul_mat_idx(up, x, idx)
        bound = (cols + 8) * 2.0 ** -24 * (xr.abs() @ U[on].abs().T)
        assert ((got[:, on].double() - (xr @ U[on].T) * keep).abs() <= bound + 1e-30).all()
        other = torch.ones(rows, dtype=torch.bool, device="cuda")
        other[on] = False
        assert not got[:, other].any()
        got = ops.sparse_ffn(up, gate if gated else None, down, x, idx).double()
        h = torch.relu(ops.ggml_mul_mat_idx(gate, x, idx)) * ops.ggml_mul_mat_idx(up, x, idx) if gated else torch.relu(ops.ggml_mul_mat_idx(up, x, idx))
        c = rounded(ops, wtype, h)[:, on] * keep
        # sums in another order (2^-22 of a hidden value) flip the rounding of one coefficient in 2^11 (FP16) or 2^15 / 127 x 64 (Q8_0: 127
        # levels), by 2^-11 of it or 2^-7 of its block's largest: 2^-11 / 45 and 2^-7 / 16 of a sum of random signs, three times over
        assert (got - c @ D[on]).norm() <= (4e-5 if wtype == synth.F16 else 2e-3) * (c @ D[on]).norm()


@pytest.mark.parametrize("T", [1, 4, 40])
def test_dense_operators_keep_a_status_word(ops, T):
    """pi_op_status finds the word of a dense product too, and it is clear: 0xFF bytes before, whatever the activations are."""
    gen = generator(T)
    x = torch.randn(T, 512, device="cuda", generator=gen)
    for wtype in (synth.F16, synth.Q4_0):
        W = weight(ops, wtype, 100, 512, gen)
        ops.ggml_mul_mat(W, x)                                        # (the workspace has its size)
        ops._ws.buf.fill_(255)
        ops.ggml_mul_mat(W, x)
        assert ops.last_op_status() == 0
    fc1, fc2 = weight(ops, synth.F16, 64, 512, gen), weight(ops, synth.F16, 300, 64, gen)
    ops._ws.buf.fill_(255)
    ops.predictor(fc1, fc2, x)
    assert ops.last_op_status() == 0


@pytest.mark.parametrize("wtype", [synth.F16, synth.Q4_0])
@pytest.mark.parametrize("T", [1, 2, 9, 40])
def test_dense_product_in_a_workspace_for_the_activations_alone(ops, wtype, T):
    """A workspace without room for control words is accepted; the kernels without waits give the same result."""
    from powerinfer_b200._lib import check, lib
    rows, cols = 333, 1024
    gen = generator(T)
    W = weight(ops, wtype, rows, cols, gen)
    x = torch.randn(T, cols, device="cuda", generator=gen)
    planes = [T * cols * 2] if wtype == synth.F16 else [T * cols // 2] * 2 + [T * cols // 8] * 2
    need = sum((b + 255) // 256 * 256 for b in planes)
    buf = torch.full((need + 512,), 255, dtype=torch.uint8, device="cuda")
    at = (-buf.data_ptr()) % 256
    out = torch.empty(T, rows, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    check(lib.pi_mul_mat(wtype, W.ptr, rows, cols, x.data_ptr(), T, None, out.data_ptr(), buf.data_ptr() + at, need, st))
    assert (buf[at + need:] == 255).all() and (buf[:at] == 255).all()
    xr, w = rounded(ops, wtype, x), ops.dequantize(W).double()
    assert ((out.double() - xr @ w.T).abs() <= (cols + 8) * 2.0 ** -24 * (xr.abs() @ w.abs().T)).all()
    assert lib.pi_mul_mat(wtype, W.ptr, rows, cols, x.data_ptr(), T, None, out.data_ptr(), buf.data_ptr() + at, need - 1, st) == 3


def test_operators_run_on_the_current_stream(ops, monkeypatch):
    """With torch's private functions, and without them."""
    side = torch.cuda.Stream()
    for names in ((), ("_raw_stream",), ("_raw_device",)):
        for name in names:
            monkeypatch.setattr(ops, name, None)
        assert ops._stream() == torch.cuda.current_stream().cuda_stream
        with torch.cuda.stream(side):
            assert ops._stream() == side.cuda_stream
        monkeypatch.undo()


@pytest.mark.parametrize("wtype", [synth.F16, synth.Q4_0])
@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("T", [32, 33, 77, 129, 256, 261])
def test_sparse_ffn_of_many_rows_per_cta(ops, wtype, gated, T):
    """Every CTA's share of the rows takes several tiles (277 neurons, 554 rows with the gate), most of them full."""
    F, d = 40960, 256
    gen = generator(T)
    up, gate, down = (weight(ops, wtype, F, d, gen) for _ in range(3))
    x = torch.randn(T, d, device="cuda", generator=gen)
    idx = torch.randn(T, F, device="cuda", generator=gen) + 0.5
    idx[:, torch.rand(F, device="cuda", generator=gen) < 0.1] = -1.0                               # active for no token
    bias = None if gated else torch.randn(F, device="cuda", generator=gen) * 0.1
    got = ops.sparse_ffn(up, gate if gated else None, down, x, idx, up_bias=bias).double()
    xr, keep = rounded(ops, wtype, x), (idx >= 0).double()
    h = xr @ ops.dequantize(up).double().T
    h = (torch.relu(xr @ ops.dequantize(gate).double().T) * h if gated else h + bias) * (keep if gated else 1.0)
    if not gated:
        h = torch.relu(torch.where(keep > 0, h, bias[None, :].double()))                            # an inactive neuron's block sees relu(bias)
    ref = (rounded(ops, wtype, h.float()) * keep) @ ops.dequantize(down).double()
    # hidden values in FP32 against float64: 2^-22 of them, which flips one rounding in 2^11 (FP16) or one of 127 levels in 2^14, each worth
    # 2^-11 or 2^-7 of a term; FP16 factors of a rounded Q4_0 sum do not occur at this width.  A missing neuron moves the sum by 1 / 200.
    assert (got - ref).norm() <= (4e-5 if wtype == synth.F16 else 1e-3) * ref.norm()


@pytest.mark.parametrize("cols", [8, 24, 56])
@pytest.mark.parametrize("T", [2, 33, 100, 200])
def test_rows_shorter_than_a_tile(ops, cols, T):
    rows = 77
    gen = generator(cols + T)
    W = weight(ops, synth.F16, rows, cols, gen)
    x = torch.randn(T, cols, device="cuda", generator=gen)
    xr, w = rounded(ops, synth.F16, x), ops.dequantize(W).double()
    bound = (cols + 8) * 2.0 ** -24 * (xr.abs() @ w.abs().T)
    assert ((ops.ggml_mul_mat(W, x).double() - xr @ w.T).abs() <= bound).all()
    idx = torch.randn(T, rows, device="cuda", generator=gen)
    assert ((ops.ggml_mul_mat_idx(W, x, idx).double() - (xr @ w.T) * (idx >= 0)).abs() <= bound).all()
    c = rounded(ops, synth.F16, torch.rand(T, rows, device="cuda", generator=gen)) * (idx >= 0)
    assert ((ops.ggml_axpy(W, c.float(), idx).double() - c @ w).abs() <= (rows + 8) * 2.0 ** -24 * (c.abs() @ w.abs())).all()


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("n_ctx", [1200, 3584, 3600])
def test_attention_of_one_token_far_into_a_sequence(ops, hd, n_ctx):
    """Positions around the ends of what a thread holds in flight (512 scores, 384 and 768 value rows), up to the last; equal scores make the
    largest sum of numerators."""
    gen = generator(hd + n_ctx)
    heads, kv = 4, 2
    kc, vc = (torch.randn(1, n_ctx, kv * hd, device="cuda", generator=gen).half() for _ in range(2))
    for pos in (0, 383, 384, 511, 512, 767, 768, 1100, n_ctx - 1):
        for scale in (1.0, 0.0):
            q = torch.randn(1, heads * hd, device="cuda", generator=gen) * scale
            k, v = (torch.randn(1, kv * hd, device="cuda", generator=gen) for _ in range(2))
            got = ops.attention_decode(q, k, v, kc, vc, torch.tensor([pos], dtype=torch.int32, device="cuda"), heads, kv)
            assert torch.equal(kc[0, pos], k[0].half()) and torch.equal(vc[0, pos], v[0].half())
            ref, bound = attention_reference(q[0], kc[0, :pos + 1], vc[0, :pos + 1], heads, kv)
            assert ((got.double().view(heads, hd) - ref).abs() <= bound).all(), (pos, scale)


@pytest.mark.parametrize("heads,kv,hd,n_ctx", [(4, 2, 128, 2500), (16, 1, 128, 1920), (16, 1, 128, 2500), (16, 1, 64, 2500), (16, 1, 128, 3700), (20, 1, 64, 2100), (12, 12, 64, 4097)])
@pytest.mark.parametrize("many", [False, True])
def test_attention_of_a_batch_in_a_long_context(ops, heads, kv, hd, n_ctx, many):
    """Scores of 16 rows fit up to 1920 (head_dim 64: 2112) positions; longer contexts, those beyond 3584, and steps whose CTAs per head and
    token all fit the SMs at once have a kernel each."""
    gen = generator(heads + n_ctx)
    T = torch.cuda.get_device_properties(0).multi_processor_count // heads + 1 if many else 3
    pos = torch.tensor([(n_ctx - 1, 700, 1300)[t % 3] for t in range(T)], dtype=torch.int32, device="cuda")
    seq = torch.arange(T, device="cuda").roll(1).int()
    kc, vc = (torch.randn(T, n_ctx, kv * hd, device="cuda", generator=gen).half() for _ in range(2))
    q = torch.randn(T, heads * hd, device="cuda", generator=gen)
    k, v = (torch.randn(T, kv * hd, device="cuda", generator=gen) for _ in range(2))
    got = ops.attention_decode(q, k, v, kc, vc, pos, heads, kv, seq=seq).double().view(T, heads, hd)
    for t in range(T):
        s, n = int(seq[t]), int(pos[t]) + 1
        assert torch.equal(kc[s, n - 1], k[t].half()) and torch.equal(vc[s, n - 1], v[t].half())
        ref, bound = attention_reference(q[t], kc[s, :n], vc[s, :n], heads, kv)
        assert ((got[t] - ref).abs() <= bound).all(), t


def test_decode_takes_ids_in_any_container(ops):
    """Lists, arrays and tensors, of the GPU too, as a whole and one by one."""
    from powerinfer_b200 import engine
    spec = synth.ModelSpec(arch=synth.ARCH_LLAMA, wtype=synth.F16, n_layer=1, d=256, n_ff=512, n_head=2, n_head_kv=2, rank=64, n_vocab=64, n_ctx=32, seed=3)
    eng = engine.DecodeEngine(spec, synth.build_model(spec), max_batch=2)
    ref = eng.decode([5, 9], [0, 3])[0].copy()
    ids, at = torch.tensor([5, 9]), torch.tensor([0, 3])
    for tokens, pos in ((np.array([5, 9]), (0, 3)), (ids, at), (ids.cuda(), at.cuda()), (list(ids), list(at)), (list(ids.cuda()), list(at.cuda())), (ids.int().cuda(), [0, 3])):
        assert np.array_equal(eng.decode(tokens, pos)[0], ref)
    eng.close()


@pytest.mark.parametrize("wtype", [synth.F16, synth.Q4_0])
@pytest.mark.parametrize("T", [1, 4, 40])
def test_operators_in_a_captured_graph(ops, wtype, T):
    """Every operator of an FFN captured behind a copy and behind another stream's work, replayed with other inputs."""
    gen = generator(T)
    F, d = 1024, 512
    up, gate, down = (weight(ops, wtype, F, d, gen) for _ in range(3))
    fc1, fc2 = weight(ops, synth.F16, 64, d, gen), weight(ops, synth.F16, F, 64, gen)
    x, src = torch.zeros(T, d, device="cuda"), torch.randn(T, d, device="cuda", generator=gen)
    bucket = torch.arange(0, 512, device="cuda", dtype=torch.int32)
    half = [weight(ops, wtype, 512, d, gen) for _ in range(2)]

    def step():
        x.copy_(src)
        idx = ops.predictor(fc1, fc2, x)
        h = torch.relu(ops.ggml_mul_mat_idx(gate, x, idx)) * ops.ggml_mul_mat_idx(up, x, idx)
        return (idx, h, ops.ggml_axpy(down, h, idx), ops.sparse_ffn(up, gate, down, x, idx), ops.ggml_mul_mat(up, x),
                ops.sparse_ffn(half[0], None, half[1], x, idx, gpu_bucket=bucket))

    eager = step()                                                    # (the workspace has its size)
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            src.mul_(1.0)
        torch.cuda.current_stream().wait_stream(side)
        captured = step()
    for scale in (1.0, -0.5):
        src.mul_(scale)
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(captured, eager if scale == 1.0 else step()):
            assert torch.equal(a, b)


def test_fewer_tokens_cost_no_more(ops):
    """2 and 8 tokens take the same instance of the same kernel, and the same bytes of weights: 2 may not take longer (they did, 1.6 times,
    when the token columns without a token were filled with copies of the last one).  The margin is for the clock of the events."""
    gen = generator(7)
    W = weight(ops, synth.Q4_0, 10240, 8192, gen)

    def best(T):
        x = torch.randn(T, 8192, device="cuda", generator=gen)
        g = torch.cuda.CUDAGraph()
        ops.ggml_mul_mat(W, x)
        torch.cuda.synchronize()
        with torch.cuda.graph(g):
            for _ in range(8):
                ops.ggml_mul_mat(W, x)
        times = []
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            g.replay()
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    two, eight = best(2), best(8)
    assert two <= 1.2 * eight, (two, eight)
