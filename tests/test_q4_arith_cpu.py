"""Arithmetic shortcuts of the Q4_0 kernels restated in numpy and checked on the CPU.  The products of several tokens (csrc/pi_mm.cu,
csrc/pi_mm_wide.cu) rely on:

* operand order: the low nibbles of a block's 16 bytes pair with Q8_0 values 0..15, the high nibbles with 16..31, and one logic
  operation makes the int8 value 16 * (q - 8) of a nibble, so that a block's integer dot is 16 times that of vec_dot_q4_0_q8_0
  (ggml-quants.c:2586-2610); scaled and summed over the blocks in FP32 it must agree with the CPU checker's mat-vec;
* the integer-to-float trick: on top of the C operand 0x4B400000 the accumulator holds the bits of the float 12582912 + 16 * dot,
  and one fused multiply-add with the block's scale dd gives 16 * dot * dd rounded once, because 12582912 * dd is exact.

The down projection (csrc/pi_axpy_mm.cu, csrc/pi_sparse.cu) makes q - 8 in FP16, BF16 and FP32 from bit patterns, and the exact mode
carries a 32-bit factor as the sum of three BF16 numbers."""
import numpy as np

from oracle import pio
from powerinfer_b200 import synth

MAGIC = 0x4B400000


def fmaf(a, b, c):
    """a * b + c for FP32 values whose product and sum fit the 64 bits of a long double, rounded once to FP32"""
    return (np.asarray(a, np.longdouble) * np.asarray(b, np.longdouble) + np.asarray(c, np.longdouble)).astype(np.float32)


def test_magic_number_conversion_is_exact_over_the_whole_range():
    q = np.arange(256, dtype=np.uint8)                                            # a byte of nibbles, as the kernels expand it
    lo, hi = (((q << 4) & 0xF0) ^ 0x80).view(np.int8), ((q & 0xF0) ^ 0x80).view(np.int8)
    assert np.array_equal(lo, 16 * ((q & 0x0F).astype(np.int32) - 8)) and np.array_equal(hi, 16 * ((q >> 4).astype(np.int32) - 8))
    dot = np.arange(-8 * 127 * 32, 8 * 127 * 32 + 1, dtype=np.int64)              # every possible block dot of q - 8 in -8..7 and int8 in -127..127
    acc = (MAGIC + 16 * dot).astype(np.uint32).view(np.float32)                   # what the integer mma leaves in the accumulator
    assert np.abs(16 * dot).max() < 2 ** 22
    assert np.array_equal(acc - np.float32(12582912.0), (16 * dot).astype(np.float32))
    # scales of the activation: FP16 numbers, the smallest subnormal and the largest among them
    rng = np.random.default_rng(0)
    for dd in [np.float32(np.float16(x)) for x in (2.0 ** -24, 6e-5, 1.0, 65504.0)] + list(np.float16(np.abs(rng.standard_normal(8)) * 0.01).astype(np.float32)):
        md = np.float32(dd * np.float32(-12582912.0))
        assert np.float64(md) == np.float64(dd) * -12582912.0                     # exact
        assert np.array_equal(fmaf(acc, dd, md), (16.0 * dot * np.float64(dd)).astype(np.float32))


def test_block_dot_operand_order_matches_the_cpu_dot():
    rng = np.random.default_rng(1)
    o = pio.Oracle()
    rows, cols, T = 24, 512, 3
    W = synth.quantize_q4_0(rng.standard_normal((rows, cols), dtype=np.float32) * np.float32(0.02))
    x = rng.standard_normal((T, cols), dtype=np.float32)
    ref = o.mul_mat(synth.Q4_0, W, rows, cols, x)                                 # CPU checker, the reference's lane order
    nb = cols // 32
    wb = W.reshape(rows, nb, 18)
    d4 = wb[:, :, :2].copy().view(np.float16).astype(np.float32)[:, :, 0]         # [rows, nb]
    qs = wb[:, :, 2:]
    lo_n, hi_n = (((qs << 4) & 0xF0) ^ 0x80).view(np.int8).astype(np.int32), ((qs & 0xF0) ^ 0x80).view(np.int8).astype(np.int32)   # values 0..15 | 16..31
    out = np.zeros((T, rows), np.float32)
    for t in range(T):
        q8 = o.quantize_q8_0(x[t]).reshape(nb, 34)
        d8 = q8[:, :2].copy().view(np.float16).astype(np.float32)[:, 0]           # [nb]
        v = q8[:, 2:].view(np.int8).astype(np.int32)                              # [nb, 32]
        dot = (lo_n * v[None, :, :16]).sum(axis=2) + (hi_n * v[None, :, 16:]).sum(axis=2)   # [rows, nb]: s8 x s8 -> s32
        c = (MAGIC + dot).astype(np.uint32).view(np.float32)
        acc = np.zeros(rows, np.float32)
        for b in range(nb):                                                       # two fused multiply-adds per block, the 1/16 in the activation's scale
            dd = np.float32(d8[b] * np.float32(0.0625))
            acc = fmaf(fmaf(c[:, b], dd, np.float32(dd * np.float32(-12582912.0))), d4[:, b], acc)
        out[t] = acc
    assert np.abs(out - ref).max() <= 2e-5, np.abs(out - ref).max()


def bf16(x):
    """round to nearest even, as cvt.rn.bf16"""
    u = np.asarray(x, np.float32).view(np.uint32)
    return ((u + 0x7FFF + ((u >> 16) & 1)) & np.uint32(0xFFFF0000)).view(np.float32)


def test_axpy_nibbles_and_split_factors():
    """csrc/pi_sparse.cu: 0x4B000000 | q is 8388608 + q.  csrc/pi_axpy_mm.cu: 0x6400 | q is the FP16 number 1024 + q, 0x6400 | q << 4 is
    1024 + 16 q, 0x4300 | q the BF16 number 128 + q; each becomes q - 8 in one exact operation.  The FP16 mode rounds weight and
    coefficient once each, 2^-10 of a term; the exact mode's three BF16 parts keep a factor to 2^-24."""
    q = np.arange(16, dtype=np.uint32)
    want = (q.astype(np.int32) - 8).astype(np.float32)
    assert np.array_equal((q | 0x4B000000).view(np.float32) - np.float32(8388616.0), want)
    half = lambda bits: np.asarray(bits, np.uint16).view(np.float16)
    assert np.array_equal(half(q | 0x6400) + half(0xE408), want.astype(np.float16))
    assert np.array_equal((half(q << 4 | 0x6400).astype(np.float64) * half(0x2C00) + np.float64(half(0xD480))).astype(np.float16), want.astype(np.float16))
    brain = lambda bits: (np.asarray(bits, np.uint32) << 16).view(np.float32)
    assert np.array_equal(bf16(brain(q | 0x4300) + brain(0xC308)), want)
    rng = np.random.default_rng(0)
    d = np.float16(np.abs(rng.standard_normal(20000)) * 0.01 + 1e-3).astype(np.float32)
    c = (rng.integers(-127, 128, d.size).astype(np.float32) * np.float16(np.abs(rng.standard_normal(d.size)) * 0.1 + 1e-3).astype(np.float32))
    qi = rng.integers(-8, 8, d.size).astype(np.float32)
    exact = qi.astype(np.float64) * d * c
    rounded = np.float16(qi * d).astype(np.float64) * np.float16(c)
    assert np.all(np.abs(rounded - exact) <= 2.0 ** -10 * np.abs(exact))
    x = c * d
    left, parts = x, []
    for _ in range(3):
        parts.append(bf16(left))
        left = left - parts[-1]                                                   # exact: the difference of neighbours
    total = sum(p.astype(np.float64) for p in parts)
    assert np.all(np.abs(total - x) <= 2.0 ** -24 * np.abs(x))
