"""The tcgen05 kernels for many tokens where they can go wrong: edges of token tiles, of row tiles and of slices of columns, ranges of few and
of many rows, no and every row active.

References are float64 sums over the values that the kernels multiply (FP16 with FP16): products are exact, so a result is off by at most
one rounding of 2^-23 per term of its sum (sums are FP32, rounded or cut)."""
import pytest

from powerinfer_b200 import synth
from test_gpu_batch_edges import generator
from test_gpu_batches import weight

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


# 38040 rows: two tiles of rows per CTA; 1184 rows: 8 per CTA; 8, 24, 520, 1032 columns: parts of a slice, of a stage of several slices
@pytest.mark.parametrize("T", [33, 128, 129, 261])
@pytest.mark.parametrize("rows,cols", [(8, 8), (1184, 1032), (3001, 520), (38040, 64)])
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
