"""The tcgen05 kernels for many tokens where they can go wrong: edges of token tiles, of row tiles and of slices of columns, ranges of few and
of many rows, no and every row active.

References are float64 sums over the values that the kernels multiply (FP16 with FP16): products are exact, so a result is off by at most
one rounding of 2^-23 per term of its sum (sums are FP32, rounded or cut)."""
import pytest

from powerinfer_b200 import synth
from test_gpu_batch_edges import generator
from test_gpu_batches import rounded, weight

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from powerinfer_b200 import ggml_ops
    return ggml_ops


def close(got, x, w, terms):
    """got = x w^T; x [T, n], w [rows, n] in float64"""
    assert ((got.double() - x @ w.T).abs() <= (terms + 4) * 2.0 ** -23 * (x.abs() @ w.abs().T) + 1e-30).all()


# 38040 rows: two tiles of rows per CTA; 1184 rows: 8 per CTA; 8, 24, 520, 1032 columns: parts of a slice, of a stage of several slices.  2048 columns and
# more, up to 5280 rows: four CTAs share the columns (33, 34 or 65 slices), clusters without rows, the line itself
@pytest.mark.parametrize("T", [33, 128, 129, 261])
@pytest.mark.parametrize("rows,cols", [(8, 8), (1184, 1032), (3001, 520), (38040, 64), (8, 2048), (1001, 2120), (5120, 2056), (5290, 2048), (2100, 4104)])
def test_dense_products(ops, rows, cols, T):
    gen = generator(rows + T)
    W, x = weight(ops, synth.F16, rows, cols, gen), torch.randn(T, cols, device="cuda", generator=gen)
    close(ops.ggml_mul_mat(W, x), x.half().double(), ops.dequantize(W).double(), cols)
    assert ops.last_op_status() == 0


@pytest.mark.parametrize("share", [0.0, 0.004, 0.6, 1.0])
@pytest.mark.parametrize("rows,cols,T", [(640, 24, 33), (5000, 1032, 77), (5000, 520, 129), (40000, 136, 40), (20000, 72, 256)])
def test_gathered_products(ops, rows, cols, T, share):
    """ggml_mul_mat_idx and the gated gather of the whole FFN: the union of the tokens' rows, zeros where a token is inactive."""
    gen = generator(rows + T)
    up, gate, down = (weight(ops, synth.F16, rows, cols, gen) for _ in range(3))
    x = torch.randn(T, cols, device="cuda", generator=gen)
    idx = torch.where((torch.rand(1, rows, device="cuda", generator=gen) < share) & (torch.rand(T, rows, device="cuda", generator=gen) < 0.7), 1.0, -1.0)
    on, xd, u = idx >= 0, x.half().double(), ops.dequantize(up).double()
    got = ops.ggml_mul_mat_idx(up, x, idx)
    assert (got[~on] == 0).all()
    ref, scale = xd @ u.T, xd.abs() @ u.abs().T
    assert ((got.double() - ref).abs() <= (cols + 4) * 2.0 ** -23 * scale + 1e-30)[on].all()
    some = torch.sort(torch.randperm(rows + 64, device="cuda", generator=gen)[:rows])[0]
    wide = torch.full((T, rows + 64), 1.0, device="cuda")
    wide[:, some] = idx
    assert torch.equal(ops.ggml_mul_mat_idx(up, x, wide, some.int(), rows + 64)[:, some], got)     # another numbering, the same sums
    g = torch.relu(ops.ggml_mul_mat_idx(gate, x, idx))
    h = (g * got).half().double() * on                                # (the FFN's hidden values are those of the two nodes)
    d = ops.dequantize(down).double()
    y = ops.sparse_ffn(up, gate, down, x, idx).double()
    assert ((y - h @ d).abs() <= (rows * share + 8) * 2.0 ** -23 * (h.abs() @ d.abs()) + 1e-30).all()
    assert ops.last_op_status() == 0


# list ranges that end inside a stage of 64, no and every row, columns in parts of a range, one accumulator and several, a second launch
@pytest.mark.parametrize("share", [0.0, 0.01, 0.7, 1.0])
@pytest.mark.parametrize("rows,cols,T", [(40, 1024, 65), (1500, 3072, 77), (3001, 2056, 129), (700, 1032, 128), (900, 520, 256), (5000, 4096, 261), (300, 8, 70)])
def test_axpy_of_many_tokens(ops, rows, cols, T, share):
    gen = generator(rows + T)
    W = weight(ops, synth.F16, rows, cols, gen)
    idx = torch.where((torch.rand(1, rows, device="cuda", generator=gen) < share) & (torch.rand(T, rows, device="cuda", generator=gen) < 0.7), 1.0, -1.0)
    h = torch.randn(T, rows, device="cuda", generator=gen).relu()
    c, w = h.half().double() * (idx >= 0), ops.dequantize(W).double()
    got = ops.ggml_axpy(W, h, idx)
    assert ((got.double() - c @ w).abs() <= (rows * share + 8) * 2.0 ** -23 * (c.abs() @ w.abs()) + 1e-30).all()
    assert torch.equal(got, ops.ggml_axpy(W, h, idx))
    assert ops.last_op_status() == 0


def test_prompt_with_rounded_factors_of_256_columns():
    """Q4_0 rows go to k_axpy_tc within prompts only, where their factors are rounded to FP16: a prompt against the same prompt token by
    token, at a width of two ranges of 256 columns and more (1024 columns, in ranges of 128: test_gpu_prefill)."""
    from powerinfer_b200 import engine
    from test_gpu_prefill import against_single_steps
    against_single_steps(engine, synth.ModelSpec(arch=synth.ARCH_LLAMA, wtype=synth.Q4_0, n_layer=1, d=2048, n_ff=5024, n_head=16, n_head_kv=4, rank=64, n_vocab=256,
                                                 n_ctx=256, firing=0.6, seed=9), (77, 129, 200))


def close_q4(got, x, w, keep=None):
    """Each product of halves is exact, the dropped ones lie below 2^-22 of their term, a drain of 64 terms is cut up to 12 times at 2^-23 of what it
    holds then, and the drains are added in FP32: within one unit of 2^-23 per 4 terms, which is asserted."""
    ref, mass = x @ w.T, x.abs() @ w.abs().T
    err = (got.double() - ref).abs()
    if keep is not None:
        err = err * keep
    assert (err <= (x.shape[1] / 4 + 16) * 2.0 ** -23 * mass + 1e-30).all()
    ref, err = (ref, err) if keep is None else (ref * keep, err)
    assert err.norm() <= 4e-7 * ref.norm() + 1e-30


# 9.. rows per CTA, tiles of 16, 96, 160 rows and several of them, sizes around every line of mm_q4_takes, a second launch
@pytest.mark.parametrize("rows,cols,T", [(8, 2048, 193), (1000, 2304, 256), (2370, 4352, 200), (10000, 2048, 97), (24000, 2048, 128), (12100, 2048, 256), (5000, 2048, 261)])
def test_q4_products(ops, rows, cols, T):
    gen = generator(rows + T)
    W, x = weight(ops, synth.Q4_0, rows, cols, gen), torch.randn(T, cols, device="cuda", generator=gen) * torch.exp(torch.randn(1, cols, device="cuda", generator=gen))
    bias = torch.randn(rows, device="cuda", generator=gen)
    got = ops.ggml_mul_mat(W, x)
    close_q4(got, rounded(ops, synth.Q4_0, x), ops.dequantize(W).double())
    assert torch.equal(ops.ggml_mul_mat(W, x, bias), got + bias)
    assert ops.last_op_status() == 0


@pytest.mark.parametrize("share", [0.0, 0.004, 0.6, 1.0])
@pytest.mark.parametrize("rows,cols,T", [(640, 2048, 97), (5000, 2304, 128), (24000, 2048, 129), (3001, 4096, 256)])
def test_q4_gathers(ops, rows, cols, T, share):
    gen = generator(rows + T)
    up, gate = weight(ops, synth.Q4_0, rows, cols, gen), weight(ops, synth.Q4_0, rows, cols, gen)
    x = torch.randn(T, cols, device="cuda", generator=gen)
    idx = torch.where((torch.rand(1, rows, device="cuda", generator=gen) < share) & (torch.rand(T, rows, device="cuda", generator=gen) < 0.7), 1.0, -1.0)
    on, xr = idx >= 0, rounded(ops, synth.Q4_0, x)
    got = ops.ggml_mul_mat_idx(up, x, idx)
    assert (got[~on] == 0).all()
    close_q4(got, xr, ops.dequantize(up).double(), on)
    if rows % 32 == 0:                                                # the gated gather of the whole FFN: its hidden values are those of the two nodes
        h, down = torch.relu(ops.ggml_mul_mat_idx(gate, x, idx)) * got, weight(ops, synth.Q4_0, rows, cols, gen)
        assert torch.equal(ops.sparse_ffn(up, gate, down, x, idx), ops.ggml_axpy(down, h, idx))
    assert ops.last_op_status() == 0


def test_q4_tokens_above_the_halves_range(ops):
    """Blocks of a token whose scale times 127 is above 65504, beside tokens and blocks with small ones."""
    rows, cols, T = 1000, 2048, 200
    gen = generator(3)
    W, x = weight(ops, synth.Q4_0, rows, cols, gen), torch.randn(T, cols, device="cuda", generator=gen)
    x[3] *= 3e4
    x[70, 64:96] *= 1e6
    x[71, ::3] *= 1e-4
    x[199] *= 2e6
    close_q4(ops.ggml_mul_mat(W, x), rounded(ops, synth.Q4_0, x), ops.dequantize(W).double())


def test_q4_rows_above_the_halves_range(ops):
    """Rows with weights above 65504, single blocks of them among others, in a dense product and a gather with gate."""
    rows, cols, T = 1024, 2048, 200
    gen = generator(4)
    w = torch.randn(rows, cols, device="cuda", generator=gen) * 0.05
    w[5] *= 2e6
    w[700, 320:352] *= 2e6
    w[1023, ::7] *= 1.5e6
    W = ops.upload_weight(synth.quantize_q4_0(w.cpu().numpy()), synth.Q4_0, rows, cols)
    x, wd = torch.randn(T, cols, device="cuda", generator=gen), ops.dequantize(W).double()
    assert (wd.abs() > 65504).any(1).sum() == 3 and wd.isfinite().all()
    close_q4(ops.ggml_mul_mat(W, x), rounded(ops, synth.Q4_0, x), wd)
    idx = torch.where(torch.rand(T, rows, device="cuda", generator=gen) < 0.7, 1.0, -1.0)
    got = ops.ggml_mul_mat_idx(W, x, idx)
    close_q4(got, rounded(ops, synth.Q4_0, x), wd, idx >= 0)
    x, down = x * 0.0001, weight(ops, synth.Q4_0, rows, cols, gen)       # (hidden values within the range of Q8_0's scales; up and gate the same rows)
    got = ops.ggml_mul_mat_idx(W, x, idx)
    y = ops.ggml_axpy(down, torch.relu(got) * got, idx)
    assert y.isfinite().all() and torch.equal(ops.sparse_ffn(W, W, down, x, idx), y)
    assert ops.last_op_status() == 0


@pytest.mark.parametrize("rows,T", [(1000, 200), (12100, 128)])
def test_q4_blocks_beside_one_above_the_halves_range(ops, rows, T):
    """Scales around 0.0002 beside scales of up to 30000 in blocks where a row's weights are 0: the result is that of the small ones alone."""
    cols, gen = 3072, generator(rows)
    raw = torch.from_numpy(synth.quantize_q4_0((torch.randn(rows, cols, device="cuda", generator=gen) * 0.05).cpu().numpy()).reshape(rows, cols // 32, 18).copy())
    raw[:, ::2, 2:] = 0x88
    W = ops.upload_weight(raw.reshape(-1).numpy(), synth.Q4_0, rows, cols)
    x = torch.randn(T, cols, device="cuda", generator=gen) * 0.01
    x.view(T, -1, 2, 32)[::3, :, 0] *= 10.0 ** (3 + 5 * torch.rand((T + 2) // 3, cols // 64, 1, device="cuda", generator=gen))
    close_q4(ops.ggml_mul_mat(W, x), rounded(ops, synth.Q4_0, x), ops.dequantize(W).double())
    idx = torch.where(torch.rand(T, rows, device="cuda", generator=gen) < 0.7, 1.0, -1.0)
    close_q4(ops.ggml_mul_mat_idx(W, x, idx), rounded(ops, synth.Q4_0, x), ops.dequantize(W).double(), idx >= 0)
    assert ops.last_op_status() == 0


def q4_of(ops, rows, cols, gen, exponents):
    """Random whole weights (-8 .. 7), a power of two as every block's scale."""
    raw = torch.randint(0, 256, (rows, cols // 32, 18), dtype=torch.uint8, device="cuda", generator=gen)
    scale = 2.0 ** torch.randint(exponents[0], exponents[1] + 1, (rows, cols // 32, 1), device="cuda", generator=gen)
    raw[..., :2] = scale.half().view(torch.uint8)
    return ops.upload_weight(raw.reshape(-1).cpu().numpy(), synth.Q4_0, rows, cols)


@pytest.mark.parametrize("rows,cols,T", [(1000, 2816, 256), (2370, 8192, 200), (12100, 3072, 128), (1000, 2048, 256)])
def test_q4_sums_that_fit_fp32_are_exact(ops, rows, cols, T):
    """Whole numbers at scales that are powers of two: a sum is a multiple of 2^-6 and stays below 2^18 (asserted of the results), so that 24 bits hold
    it at every step: nothing may be cut or rounded."""
    gen = generator(rows)
    W = q4_of(ops, rows, cols, gen, (-6, -2))
    x = torch.randint(-20, 21, (T, cols), device="cuda", generator=gen).float()
    x[:, ::32] = 127.0                                                # (a block's largest value: scales of 1)
    ref = x.double() @ ops.dequantize(W).double().T
    assert ref.abs().max() < 2.0 ** 18 and torch.equal(rounded(ops, synth.Q4_0, x), x.double())
    assert torch.equal(ops.ggml_mul_mat(W, x).double(), ref)
    idx = torch.where(torch.rand(T, rows, device="cuda", generator=gen) < 0.7, 1.0, -1.0)
    assert torch.equal(ops.ggml_mul_mat_idx(W, x, idx).double(), ref * (idx >= 0))


@pytest.mark.parametrize("rows,cols,T", [(1000, 2816, 256), (12100, 8192, 128)])
def test_q4_tokens_of_one_feature(ops, rows, cols, T):
    """One term: the product of the rests, 2^-22 of it, is left out, and the others are cut once each at 2^-23 of their sum."""
    gen = generator(cols)
    W, x = weight(ops, synth.Q4_0, rows, cols, gen), torch.zeros(T, cols, device="cuda")
    x[torch.arange(T, device="cuda"), torch.randint(0, cols, (T,), device="cuda", generator=gen)] = torch.randn(T, device="cuda", generator=gen)
    ref = rounded(ops, synth.Q4_0, x) @ ops.dequantize(W).double().T
    err = (ops.ggml_mul_mat(W, x).double() - ref).abs()
    assert (err <= (2.0 ** -22 + 2 * 2.0 ** -23) * ref.abs() + 1e-30).all()
    assert err.norm() <= 7e-8 * ref.norm()


def test_q4_products_take_no_notice_of_what_tensor_memory_held(ops):
    """Ranges of 144 rows are read from tensor memory in pieces of 80 columns, so that 8 of the last piece are an earlier kernel's.  Infinite sums
    there started a search through the scales of all rows: the same product after infinite and after finite ones takes the same time."""
    sms, cols, T = torch.cuda.get_device_properties(0).multi_processor_count, 2816, 128
    gen = generator(11)
    raw = torch.randint(0, 256, (sms * 160, cols // 32, 18), dtype=torch.uint8, device="cuda", generator=gen)
    x, ws = torch.randn(T, cols, device="cuda", generator=gen), []
    for scale, rows in ((float("inf"), 160), (0.01, 160), (0.01, 144)):
        raw[..., :2] = torch.full((1, 1, 1), scale, device="cuda").half().view(torch.uint8)
        ws.append(ops.upload_weight(raw[:sms * rows].reshape(-1).cpu().numpy(), synth.Q4_0, sms * rows, cols))
    times = []
    for before in ws[:2] * 5:
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ops.ggml_mul_mat(before, x)
        a.record()
        y = ops.ggml_mul_mat(ws[2], x)
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b))
        assert y.isfinite().all()
    assert min(times[0::2]) < 1.3 * min(times[1::2]), times


@pytest.mark.parametrize("more", [0, 1])
@pytest.mark.parametrize("share", [80, 96])
def test_q4_products_around_one_tile_a_cta(ops, share, more):
    """Rows on both sides of the lines between k_mm_q4 (one tile, several) and k_mm_wide (two tiles there, one here)."""
    rows, cols, T = torch.cuda.get_device_properties(0).multi_processor_count * share + more, 2816, 200
    gen = generator(rows)
    W, x = weight(ops, synth.Q4_0, rows, cols, gen), torch.randn(T, cols, device="cuda", generator=gen)
    close_q4(ops.ggml_mul_mat(W, x), rounded(ops, synth.Q4_0, x), ops.dequantize(W).double())
    assert ops.last_op_status() == 0


# ---- the same at sizes that take other paths today.  Short rows: two and three slices, all in one stage
@pytest.mark.parametrize("T", [33, 128, 129, 261])
@pytest.mark.parametrize("rows,cols", [(700, 136), (9001, 192), (300, 72)])
def test_dense_products_of_short_rows(ops, rows, cols, T):
    test_dense_products(ops, rows, cols, T)


# (below 2816 columns: k_mm_wide)
@pytest.mark.parametrize("rows,cols,T", [(8, 2816, 193), (1000, 3072, 256), (10000, 2816, 97), (24000, 2816, 128), (12100, 3072, 256), (5000, 2816, 261), (5000, 2560, 200)])
def test_q4_products_of_2816_columns_and_more(ops, rows, cols, T):
    test_q4_products(ops, rows, cols, T)


@pytest.mark.parametrize("share", [0.0, 0.004, 0.6, 1.0])
@pytest.mark.parametrize("rows,cols,T", [(640, 2816, 97), (5000, 3072, 128), (24000, 2816, 129)])
def test_q4_gathers_of_2816_columns_and_more(ops, rows, cols, T, share):
    test_q4_gathers(ops, rows, cols, T, share)


def test_wide_q4_tokens_above_the_halves_range(ops):
    """test_q4_tokens_above_the_halves_range at a width of k_mm_q4."""
    rows, cols, T = 1000, 3072, 200
    gen = generator(3)
    W, x = weight(ops, synth.Q4_0, rows, cols, gen), torch.randn(T, cols, device="cuda", generator=gen)
    x[3] *= 3e4
    x[70, 64:96] *= 1e6
    x[71, ::3] *= 1e-4
    x[199] *= 2e6
    close_q4(ops.ggml_mul_mat(W, x), rounded(ops, synth.Q4_0, x), ops.dequantize(W).double())


@pytest.mark.parametrize("T", [97, 200])
def test_wide_q4_rows_above_the_halves_range(ops, T):
    """test_q4_rows_above_the_halves_range at a width of k_mm_q4; the FFN with gate, and without it but with a bias: the sums of such rows, made anew,
    take the same epilogue."""
    rows, cols = 1024, 3072
    gen = generator(4)
    w = torch.randn(rows, cols, device="cuda", generator=gen) * 0.05
    w[5] *= 2e6
    w[700, 320:352] *= 2e6
    w[1023, ::7] *= 1.5e6
    W = ops.upload_weight(synth.quantize_q4_0(w.cpu().numpy()), synth.Q4_0, rows, cols)
    x, wd = torch.randn(T, cols, device="cuda", generator=gen), ops.dequantize(W).double()
    assert (wd.abs() > 65504).any(1).sum() == 3 and wd.isfinite().all()
    close_q4(ops.ggml_mul_mat(W, x), rounded(ops, synth.Q4_0, x), wd)
    idx = torch.where(torch.rand(T, rows, device="cuda", generator=gen) < 0.7, 1.0, -1.0)
    idx[:, 64:200] = -1.0                                             # active for no token
    close_q4(ops.ggml_mul_mat_idx(W, x, idx), rounded(ops, synth.Q4_0, x), wd, idx >= 0)
    x, down = x * 0.0001, weight(ops, synth.Q4_0, rows, cols, gen)       # (hidden values within the range of Q8_0's scales; up and gate the same rows)
    got = ops.ggml_mul_mat_idx(W, x, idx)
    close_q4(got, rounded(ops, synth.Q4_0, x), wd, idx >= 0)
    y = ops.ggml_axpy(down, torch.relu(got) * got, idx)
    assert y.isfinite().all() and torch.equal(ops.sparse_ffn(W, W, down, x, idx), y)
    bias = torch.randn(rows, device="cuda", generator=gen)
    y = ops.ggml_axpy(down, torch.relu(got + bias), idx)
    assert y.isfinite().all() and torch.equal(ops.sparse_ffn(W, None, down, x, idx, up_bias=bias), y)
    assert ops.last_op_status() == 0


def within_steps(got, ref, terms):
    """The error of a whole result, as a 2-norm: the tensor cores cut a sum at every step of 16 terms, each time by at most 2^-23 of what it holds
    then, which in the mean over the results is no more than the result itself; 20 more for partial sums added in FP32.  (Partial sums passed on
    in FP16 would be 2^-13 of the results off, four to a hundred times this.)"""
    assert (got.double() - ref).norm() <= (terms / 16 + 20) * 2.0 ** -23 * ref.norm()


# one chain, two tiles, chains in a cluster of four (2048 columns and more)
@pytest.mark.parametrize("rows,cols,T", [(300, 72, 33), (38040, 64, 128), (1184, 1032, 77), (1001, 2120, 261), (5290, 2048, 128), (2100, 4104, 77), (512, 4096, 256)])
def test_dense_products_keep_fp32_sums(ops, rows, cols, T):
    gen = generator(rows + T)
    W, x = weight(ops, synth.F16, rows, cols, gen), torch.randn(T, cols, device="cuda", generator=gen)
    within_steps(ops.ggml_mul_mat(W, x), x.half().double() @ ops.dequantize(W).double().T, cols)
    idx = torch.where(torch.rand(T, rows, device="cuda", generator=gen) < 0.6, 1.0, -1.0)
    within_steps(ops.ggml_mul_mat_idx(W, x, idx), (x.half().double() @ ops.dequantize(W).double().T) * (idx >= 0), cols)


# one accumulator and several, list ranges of one stage and of many
@pytest.mark.parametrize("share", [0.05, 0.7])
@pytest.mark.parametrize("rows,cols,T", [(1500, 3072, 77), (3001, 2056, 129), (900, 520, 256), (5000, 4096, 256)])
def test_axpy_of_many_tokens_keeps_fp32_sums(ops, rows, cols, T, share):
    gen = generator(rows + T)
    W = weight(ops, synth.F16, rows, cols, gen)
    idx = torch.where((torch.rand(1, rows, device="cuda", generator=gen) < share) & (torch.rand(T, rows, device="cuda", generator=gen) < 0.7), 1.0, -1.0)
    h = torch.randn(T, rows, device="cuda", generator=gen)
    within_steps(ops.ggml_axpy(W, h, idx), (h.half().double() * (idx >= 0)) @ ops.dequantize(W).double(), rows * share)
