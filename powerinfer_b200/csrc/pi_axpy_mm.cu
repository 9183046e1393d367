// ggml_axpy for 2 and more tokens on the tensor cores (ggml.c:14314-14618 is the CPU path it matches), and the coefficients it reads.
//
// dst[t, c] = sum over listed rows r of coef[t, r] * Wt[r, c].  As a matrix product C[c, t] += A[c, r] * B[r, t]: A = the rows
// of down_t read transposed, B = the coefficients, laid out by list position so that they load like a matrix.
//   FP16 rows: coef = FP16(h) of a token's active rows, else 0; the products of two halves are exact, sums are FP32, as on
//              the CPU.
//   Q4_0 rows, rounded: weight FP16(d * (q - 8)) (one rounding: q - 8 is exact), coef = FP16(b8 * d8) of the CPU path's int8 x
//              scale pair: two roundings to 11 bits that the CPU path does not have, relative error up to 2^-10 per term.
//   Q4_0 rows, exact: A = q - 8 (an integer, exact in BF16), B = b8 * d8 * d of a column block as the sum of
//              three BF16 numbers (24 bits, FP32's exponent range): three mma for one.  axpy_mm_exact says which.
// The nibbles become fragments in registers: a lane takes the same 4-byte word of two neighbouring rows, and one byte permute
// and one logic operation make the pair {1024 + q of row r, 1024 + q of row r + 1} of a column, in the fragment's k order.
// (Expanding a stage into an FP16 tile in shared memory first costs two barriers per 16 rows: 159 us where this takes 82,
// 103 MB of rows, 32 tokens.)
//
// Work split: units of 256 columns x 64 (128) list rows x up to 64 tokens, numbered slice by slice (a slice: 256 columns of one group of
// tokens, equal groups: fragments are expanded once for all tokens of a group, 256 tokens of 70B shape in groups of 32 took 454 us where 64 take 355; the groups of a column range follow one another, so that they find its rows in L2); every CTA takes an equal contiguous
// range, so the chip is full whatever the number of columns.  The CTAs that meet in a slice each write one partial vector
// ("piece"); at most n_pieces of them per slice, the missing ones are written as zeros, and the norm (or the reduction)
// that follows adds the pieces in order.  Rows arrive by 16-byte cp.async (they lie anywhere) from 8 producer warps; 8 consumer warps
// share a stage, 4 along the columns and 2 along the rows, and meet at the end of a slice only.  (When all 16 warps did both, a stage
// took 5500 clocks, of which its bytes need 1400: divisions for the unit's place, copies that wait while the queue of outstanding
// loads is full, a barrier.)  Every wait is bounded: when one runs out bit 4 of *status is set (where given) and the rest of the work
// is passed over.
#include "pi_common.cuh"

namespace pi {

static constexpr int AX_THREADS = 512, AX_CONS = 8, AX_PROD = 256, AX_CW = 256;      // warps 0 .. 7 consume, threads 256 .. 511 produce; columns of a unit
static constexpr int AX_SMAX = 8;                        // stages at most
static constexpr int AX_REGS_C = 200, AX_REGS_P = 56;    // 256 x (200 + 56) = the 512 x 128 of the launch
static constexpr int AX_RED_PITCH = AX_CW + 4;           // conflict-free fragment stores
static constexpr size_t AX_SMEM_MAX = 226 * 1024;

struct AxpyMmP {
    const uint8_t * Wt; int64_t row_bytes; int nrows, ncols, nb, T;
    const int32_t * list; const int32_t * count;
    const void * coef; int64_t coef_stride;                           // FP16, or F32 in the exact mode
    unsigned int * status;
    float * partial; int n_cs, n_tg, n_pieces;                        // column ranges, token groups, partial vectors per slice
};

__device__ __forceinline__ void ax_cp16(uint32_t dst, const void * src, unsigned bytes) {       // the first `bytes` bytes, the rest zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ax_ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ax_ldsm4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ax_ldsm2(uint32_t & r0, uint32_t & r1, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(addr));
}
__device__ __forceinline__ void ax_hmma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ax_bmma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t ax_bf2(float lo, float hi) { uint32_t r; asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo)); return r; }
__device__ __forceinline__ uint32_t ax_badd2(uint32_t a, uint32_t b) { uint32_t r; asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
// {x, y} as the sum of three pairs of BF16 numbers (each difference is exact in FP32)
__device__ __forceinline__ void ax_split3(float x, float y, uint32_t (&b)[3]) {
#pragma unroll
    for (int i = 0; i < 3; i++) {
        b[i] = ax_bf2(x, y);
        x -= __uint_as_float(b[i] << 16);
        y -= __uint_as_float(b[i] & 0xFFFF0000u);
    }
}
__device__ __forceinline__ uint32_t ax_mul2(uint32_t a, uint32_t b) { uint32_t r; asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ uint32_t ax_add2(uint32_t a, uint32_t b) { uint32_t r; asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ uint32_t ax_fma2(uint32_t a, uint32_t b, uint32_t c) { uint32_t r; asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c)); return r; }

enum { AX_F16 = 0, AX_Q4 = 1, AX_Q4_EXACT = 2 };

template <int MODE, int NT>
struct AxShape {
    static constexpr bool Q4 = MODE != AX_F16, EXACT = MODE == AX_Q4_EXACT;
    static constexpr int TP = NT * 8;
    static constexpr int RS = MODE == AX_Q4 ? 128 : 64;               // list rows of a stage
    static constexpr int W_PITCH = Q4 ? 144 : AX_CW * 2 + 16;         // odd multiples of 16 bytes
    static constexpr int CB = EXACT ? 4 : 2;                          // bytes of a coefficient
    static constexpr int C_PITCH = RS * CB + (EXACT ? 32 : 16);
    static constexpr int C_OFF = RS * W_PITCH;
    static constexpr int STAGE = (C_OFF + TP * C_PITCH + 127) / 128 * 128;
    static constexpr int RED = TP * AX_RED_PITCH * 4;
    static constexpr int HEAD = (RED + 127) / 128 * 128;
    static constexpr int FIT = (int)((AX_SMEM_MAX - HEAD) / STAGE);
    static constexpr int S = FIT > AX_SMAX ? AX_SMAX : FIT;
    static constexpr int KPW = RS / 32;                               // 16-row steps of a warp per stage (2 warps share the rows)
    static_assert(S >= 3, "ring");
};

template <int MODE, int NT>
__global__ void __launch_bounds__(AX_THREADS, 1) k_axpy_mm(const AxpyMmP p) {
    using Z = AxShape<MODE, NT>;
    constexpr bool Q4 = Z::Q4, EXACT = Z::EXACT;
    constexpr int TP = Z::TP, RS = Z::RS, S = Z::S, KPW = Z::KPW;
    extern __shared__ __align__(128) unsigned char smem[];
    float * red = reinterpret_cast<float *>(smem);                    // [TP][AX_RED_PITCH]
    __shared__ uint64_t s_full[AX_SMAX], s_empty[AX_SMAX];
    __shared__ volatile int s_dead;
    const uint32_t ring_a = smem_u32(smem + Z::HEAD);
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);    // (uniform for the compiler)
    const int wc = warp & 3, wk = (warp >> 2) & 1;                    // consumers: 64 columns, a half of the stage's rows
    const int cta = blockIdx.x;

    if (tid < AX_SMAX) { mbar_init(s_full + tid, AX_PROD); mbar_init(s_empty + tid, AX_CONS); }
    if (tid == 0) s_dead = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncthreads();
    auto wait = [&](uint64_t * bar, unsigned parity) -> bool {        // warp-uniform; false: the wait ran out, here or elsewhere
        bool ok = false;
        for (int spins = 0; spins < (1 << 20) && !ok && !s_dead; spins++) ok = mbar_try_wait(bar, parity);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok && lane == 0) { s_dead = 1; if (p.status) atomicOr(p.status, 16u); }
        return ok;
    };
    pdl_launch();
    pdl_wait();
    const int n = min(*p.count, p.nrows);
    const int nst = (n + RS - 1) / RS;
    const int n_sl = p.n_cs * p.n_tg;
    const unsigned total = (unsigned)n_sl * (unsigned)nst;
    if (total == 0) {                                                 // no active row: the result is zero
        for (int cs = cta; cs < p.n_cs; cs += gridDim.x)
            for (int e = tid; e < p.n_pieces * p.T * AX_CW; e += AX_THREADS) {
                const int c = cs * AX_CW + e % AX_CW;
                if (c < p.ncols) p.partial[(size_t)(e / AX_CW) * p.ncols + c] = 0.f;
            }
        return;
    }
    const unsigned G = min((unsigned)gridDim.x, total);               // every CTA that takes part has a unit
    if ((unsigned)cta >= G) return;
    const int u0 = (int)((unsigned long long)total * (unsigned)cta / G), n_units = (int)((unsigned long long)total * (unsigned)(cta + 1) / G) - u0;

    // place of the current unit: stage of the slice, slice, its column range and token group
    int st = u0 % nst, sl = u0 / nst, cs = sl / p.n_tg, tg = sl % p.n_tg;
    auto advance = [&]() {
        if (++st < nst) return;
        st = 0; sl++;
        if (++tg == p.n_tg) { tg = 0; cs++; }
    };

    if (warp >= AX_CONS) {
        // ================================================================= producers: a row of the stage per TR threads
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" :: "n"(AX_REGS_P));
        const int pt = tid - AX_CONS * 32;
        constexpr int TR = AX_PROD / RS, PW = (Q4 ? 8 : 32) / TR;      // 16-byte pieces of a row slice per thread
        const int r = pt / TR, c0 = pt % TR;
        constexpr int CPP = 16 / Z::CB, CPR = RS / CPP;               // coefficients of a 16-byte piece; pieces of a token
        constexpr int NC = (TP * CPR + AX_PROD - 1) / AX_PROD;
        auto row_at = [&](int s) {                                    // row number of my list entry in stage s of the slice
            const int v = s * RS + r < n ? p.list[s * RS + r] : 0;
            return (unsigned)v < (unsigned)p.nrows ? v : 0;
        };
        int slot = 0, row = row_at(st);
        unsigned phase = 1u;                                          // parity of the hand-back to wait for (first round: none)
        for (int i = 0; i < n_units; i++) {
            const int next_row = row_at(st + 1 < nst ? st + 1 : 0);   // (one unit ahead: its latency passes while this unit is copied)
            if (!wait(s_empty + slot, phase)) break;
            const uint32_t base = ring_a + (uint32_t)(slot * Z::STAGE);
            const bool live = st * RS + r < n;
            const uint8_t * src = p.Wt + (size_t)row * p.row_bytes;
            if (!Q4) {
                const int col = cs * AX_CW + c0 * 8;
                const uint8_t * at = src + (size_t)col * 2;
#pragma unroll
                for (int j = 0; j < PW; j++) {                        // (rows past the list: coefficients 0, but what they meet must be finite)
                    const bool ok = live && col + j * TR * 8 < p.ncols;
                    ax_cp16(base + r * Z::W_PITCH + (c0 + j * TR) * 16, ok ? at + j * TR * 16 : p.Wt, ok ? 16u : 0u);
                }
            } else {
                const uint8_t * at = src + (size_t)cs * 128 + c0 * 16;
#pragma unroll
                for (int j = 0; j < PW; j++) ax_cp16(base + r * Z::W_PITCH + (c0 + j * TR) * 16, at + j * TR * 16, live ? 16u : 0u);
                if (c0 == 0) ax_cp16(base + r * Z::W_PITCH + 128, src + (size_t)p.nb * 16 + (size_t)cs * 16, live ? 16u : 0u);
            }
            const int tok0 = tg * TP, Tg = min(TP, p.T - tok0);
#pragma unroll
            for (int j = 0; j < NC; j++) {                            // coefficients; positions past the list count as 0
                const int e = pt + j * AX_PROD, t = e / CPR, c = e % CPR, li = st * RS + c * CPP;
                if (t >= TP) break;
                const int bytes = t < Tg ? max(0, min(CPP, n - li)) * Z::CB : 0;
                ax_cp16(base + Z::C_OFF + t * Z::C_PITCH + c * 16, (const char *)p.coef + (bytes ? ((size_t)(tok0 + t) * p.coef_stride + li) * Z::CB : 0), (unsigned)bytes);
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" :: "r"(smem_u32(s_full + slot)) : "memory");
            row = next_row;
            advance();
            if (++slot == S) { slot = 0; phase ^= 1u; }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        return;
    }
    // ===================================================================== consumers
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" :: "n"(AX_REGS_C));
    float acc[4][NT][4];
    auto clear = [&]() {
#pragma unroll
        for (int m = 0; m < 4; m++)
#pragma unroll
            for (int t = 0; t < NT; t++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[m][t][j] = 0.f;
    };
    clear();
    const int g = lane >> 2, q = lane & 3, j8 = lane >> 3;
    // FP16: transposed 8x8 loads (k = list rows, m = columns).  Q4_0: word g of the warp's 64 columns, rows 2q, 2q + 1 (and + 8)
    const uint32_t a_off = Q4 ? (uint32_t)((wk * KPW * 16 + 2 * q) * Z::W_PITCH + wc * 32 + g * 4)
                              : (uint32_t)((wk * KPW * 16 + (j8 >> 1) * 8 + (lane & 7)) * Z::W_PITCH + (wc * 64 + (j8 & 1) * 8) * 2);
    const uint32_t s_off = (uint32_t)((wk * KPW * 16 + 2 * q) * Z::W_PITCH + 128 + (wc * 2 + (g >> 2)) * 2);
    const uint32_t b_off = (uint32_t)(Z::C_OFF + ((lane & 7) + (NT > 1 ? ((lane >> 4) & 1) * 8 : 0)) * Z::C_PITCH + (wk * KPW * 16 + ((lane >> 3) & 1) * 8) * 2);

    int slot = 0;
    unsigned phase = 0u;
    bool ok = true;                                                   // (when a wait ran out the barriers below are still met)
    for (int i = 0; i < n_units; i++) {
        ok = ok && wait(s_full + slot, phase);
        const uint32_t base = ring_a + (uint32_t)(slot * Z::STAGE);
        if (ok)
#pragma unroll
        for (int k = 0; k < KPW; k++) {
            if (EXACT) {
                // lane: bytes 2 * (g & 1) and the next of word g >> 1 of a block, so that an mma's rows lie in ONE column block
                // and the block's scales can go into its B operand
#pragma unroll
                for (int bl = 0; bl < 2; bl++) {
                    uint32_t w[4];
                    float d[4];
#pragma unroll
                    for (int h = 0; h < 4; h++) {
                        const uint32_t at = base + (uint32_t)(((wk * KPW + k) * 16 + 2 * q + (h >> 1) * 8 + (h & 1)) * Z::W_PITCH);
                        unsigned short x;
                        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[h]) : "r"(at + (wc * 2 + bl) * 16 + (g >> 1) * 4));
                        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(x) : "r"(at + 128 + (wc * 2 + bl) * 2));
                        d[h] = __half2float(__ushort_as_half(x));
                    }
                    uint32_t a[2][4];                                 // (bit patterns: 0x4300 = 128, 0xC308 = -136)
#pragma unroll
                    for (int m = 0; m < 2; m++) {
                        const unsigned sel = 0x4400u + 0x1111u * (unsigned)(2 * (g & 1) + m);
                        const uint32_t x = __byte_perm(w[0], w[1], sel), y = __byte_perm(w[2], w[3], sel);
                        a[m][0] = ax_badd2((x & 0x000F000Fu) | 0x43004300u, 0xC308C308u);
                        a[m][1] = ax_badd2(((x >> 4) & 0x000F000Fu) | 0x43004300u, 0xC308C308u);
                        a[m][2] = ax_badd2((y & 0x000F000Fu) | 0x43004300u, 0xC308C308u);
                        a[m][3] = ax_badd2(((y >> 4) & 0x000F000Fu) | 0x43004300u, 0xC308C308u);
                    }
#pragma unroll
                    for (int t = 0; t < NT; t++) {
                        const uint32_t at = base + (uint32_t)(Z::C_OFF + (t * 8 + g) * Z::C_PITCH + ((wk * KPW + k) * 16 + 2 * q) * 4);
                        float c[4];
                        asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(c[0]), "=f"(c[1]) : "r"(at));
                        asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(c[2]), "=f"(c[3]) : "r"(at + 32));
                        uint32_t b0[3], b1[3];
                        ax_split3(c[0] * d[0], c[1] * d[1], b0);
                        ax_split3(c[2] * d[2], c[3] * d[3], b1);
#pragma unroll
                        for (int m = 0; m < 2; m++)
#pragma unroll
                            for (int i3 = 0; i3 < 3; i3++) ax_bmma(acc[bl * 2 + m][t], a[m], b0[i3], b1[i3]);
                    }
                }
                continue;
            }
            uint32_t b[NT][2];
            if (NT == 1) ax_ldsm2(b[0][0], b[0][1], base + b_off + k * 32);
            else {
#pragma unroll
                for (int t = 0; t < NT; t += 2) {
                    uint32_t v[4];
                    ax_ldsm4(v, base + b_off + t * 8 * Z::C_PITCH + k * 32 - (t + 1 < NT ? 0u : ((lane >> 4) & 1) * 8 * Z::C_PITCH));   // (an odd last group is read twice)
                    b[t][0] = v[0]; b[t][1] = v[1];
                    if (t + 1 < NT) { b[(t + 1) % NT][0] = v[2]; b[(t + 1) % NT][1] = v[3]; }
                }
            }
            if (!Q4) {
#pragma unroll
                for (int m = 0; m < 4; m++) {
                    uint32_t a[4];
                    ax_ldsm4_trans(a, base + a_off + k * 16 * Z::W_PITCH + m * 32);
#pragma unroll
                    for (int t = 0; t < NT; t++) ax_hmma(acc[m][t], a, b[t][0], b[t][1]);
                }
            } else {
                uint32_t w[4], sc[2];
#pragma unroll
                for (int h = 0; h < 4; h++)
                    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[h]) : "r"(base + a_off + (k * 16 + (h >> 1) * 8 + (h & 1)) * Z::W_PITCH));
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    unsigned short x, y;
                    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(x) : "r"(base + s_off + (k * 16 + h * 8) * Z::W_PITCH));
                    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(y) : "r"(base + s_off + (k * 16 + h * 8 + 1) * Z::W_PITCH));
                    sc[h] = (uint32_t)x | ((uint32_t)y << 16);
                }
#pragma unroll
                for (int j = 0; j < 4; j++) {                         // byte j of the word: columns j (low nibble) and 16 + j (high)
                    const unsigned sel = 0x4400u + 0x1111u * (unsigned)j;
                    const uint32_t x = __byte_perm(w[0], w[1], sel), y = __byte_perm(w[2], w[3], sel);
                    uint32_t a[4];                                    // (bit patterns: 0x6400 = 1024, 0x2C00 = 1/16, 0xE408 = -1032, 0xD480 = -72)
                    a[0] = ax_mul2(ax_add2((x & 0x000F000Fu) | 0x64006400u, 0xE408E408u), sc[0]);
                    a[1] = ax_mul2(ax_fma2((x & 0x00F000F0u) | 0x64006400u, 0x2C002C00u, 0xD480D480u), sc[0]);
                    a[2] = ax_mul2(ax_add2((y & 0x000F000Fu) | 0x64006400u, 0xE408E408u), sc[1]);
                    a[3] = ax_mul2(ax_fma2((y & 0x00F000F0u) | 0x64006400u, 0x2C002C00u, 0xD480D480u), sc[1]);
#pragma unroll
                    for (int t = 0; t < NT; t++) ax_hmma(acc[j][t], a, b[t][0], b[t][1]);
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(s_empty + slot);                   // handed back
        if (++slot == S) { slot = 0; phase ^= 1u; }
        if (st == nst - 1 || i == n_units - 1) {
            // ---- end of this CTA's share of the slice: the row halves are added in order
            const int tok0 = tg * TP, Tg = min(TP, p.T - tok0);
#pragma unroll 1
            for (int r = 0; r < 2; r++) {
                if (wk == r) {
#pragma unroll
                    for (int m = 0; m < 4; m++)
#pragma unroll
                        for (int t = 0; t < NT; t++)
#pragma unroll
                            for (int j = 0; j < 4; j++) {
                                // fragment row g (j < 2) or g + 8: FP16: column m * 16 + that; Q4_0: word g, byte m, nibble j >> 1;
                                // exact: block m >> 1, word g >> 1, byte 2 * (g & 1) + (m & 1), nibble j >> 1
                                const int c = wc * 64 + (EXACT ? (m >> 1) * 32 + (g >> 1) * 4 + 2 * (g & 1) + (m & 1) + (j >> 1) * 16
                                                         : Q4 ? (g >> 2) * 32 + (g & 3) * 4 + m + (j >> 1) * 16 : m * 16 + g + (j >> 1) * 8);
                                float * o = red + (t * 8 + 2 * q + (j & 1)) * AX_RED_PITCH + c;
                                *o = r == 0 ? acc[m][t][j] : *o + acc[m][t][j];
                            }
                }
                asm volatile("bar.sync 1, 256;" ::: "memory");
            }
            const int c_lo = (int)((((unsigned long long)sl * nst + 1u) * G - 1u) / total), c_hi = (int)(((unsigned long long)(sl + 1) * nst * G - 1u) / total);
            const int piece = cta - c_lo, more = cta == c_hi ? p.n_pieces - 1 - piece : 0;      // the slice's last CTA also writes the missing pieces
            for (int e = tid; e < Tg * AX_CW; e += AX_CONS * 32) {
                const int c = e % AX_CW, t = e / AX_CW, col = cs * AX_CW + c;
                if (col >= p.ncols) continue;
                float * o = p.partial + ((size_t)piece * p.T + tok0 + t) * p.ncols + col;
                *o = red[t * AX_RED_PITCH + c];
                for (int k = 1; k <= more; k++) o[(size_t)k * p.T * p.ncols] = 0.f;
            }
            clear();
            asm volatile("bar.sync 1, 256;" ::: "memory");             // the sums are read
        }
        advance();
    }
}

// ---------------------------------------------------------------------------------------------- coefficients
// h F32 [T, h_stride] (by global neuron id) -> coef [T, coef_stride] by list position: FP16(h), or for Q4_0 rows the int8
// quant of h in its block of 32 neurons times that block's FP16 scale (ggml.c:14575-14581, quantize_row_q8_0), rounded to FP16
// or (exact mode) as it is, in F32; 0 where the token is inactive.  The block is the one of the GLOBAL ids.  Where a warp's rows are one
// whole block (always without a bucket) its maximum is the warp's; any other bucket's rows read their blocks from h, which then holds
// something at every neuron (BLOCKS: an instance of its own; in one kernel the look-up cost the calls that have no use for it 3 us).  One warp per 32 local rows (one word of the union masks); a
// CTA takes 8 tokens, counts the rows named by the words before its own to find its list positions, and writes its part of the list.
// Bound: the latency from the wait to the stores.  The hidden values are loaded before the count, whether the word names a row or
// not, the count meets at one barrier, and the eight tokens' maxima and quotients run side by side: eight tokens, 28672 rows, 3 layers
// 556 -> 543 us per pass; 16 tokens, 13824 rows 77.0 -> 73.5 us; 256 tokens, 28672 rows, 3 layers 5143 -> 5116 us.  (CTAs with several
// groups of 8 tokens, which count once, took 5150 .. 5200 us.)
struct CoefP {
    const float * h; int64_t h_stride; const float * idx; int64_t idx_stride; float threshold;
    const int32_t * bucket; const uint32_t * masks; int32_t * list; int32_t * count; int n_local, T;
    const float * fill_bias;
    void * coef; int64_t coef_stride; int exact;
};

template <bool Q4, bool BLOCKS>
__global__ void __launch_bounds__(256) k_coef(const CoefP p) {
    __shared__ int s_pre[8], s_cnt[8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_chunks = (p.n_local + 31) / 32;
    const int c = blockIdx.x * 8 + warp, r = c * 32 + lane;
    const bool in = r < p.n_local;
    const int64_t g = in ? (p.bucket ? p.bucket[r] : r) : 0;
    const float fill = Q4 && !BLOCKS && p.fill_bias && in ? fmaxf(p.fill_bias[g], 0.f) : 0.f;
    constexpr int UN = 8;
    pdl_launch();
    pdl_wait();
    uint32_t m = c < n_chunks ? __ldcg(p.masks + c) : 0u;
    const int t0 = blockIdx.y * UN;
    // (lanes past the last row stand for the rest of its block, which counts where h holds something there)
    const int64_t first = __shfl_sync(0xffffffffu, g, 0);
    const bool whole = !BLOCKS || __all_sync(0xffffffffu, (first & 31) == 0 && (!in || g == first + lane));
    float v[UN], l[UN];                                               // (on their way while the positions are counted)
#pragma unroll
    for (int u = 0; u < UN; u++) {
        v[u] = 0.f; l[u] = 0.f;
        if (in && t0 + u < p.T) { v[u] = p.h[(size_t)(t0 + u) * p.h_stride + g]; l[u] = p.idx[(size_t)(t0 + u) * p.idx_stride + g]; }
        if (BLOCKS && whole && !in && c < n_chunks && t0 + u < p.T) v[u] = p.h[(size_t)(t0 + u) * p.h_stride + first + lane];
    }
    int sum = 0;
#pragma unroll 4
    for (int k = tid; k < (int)blockIdx.x * 8; k += 256) sum += __popc(__ldcg(p.masks + k));
    const int left = p.n_local - c * 32;                              // bits beyond the last row never count
    if (left < 32) m &= left <= 0 ? 0u : (1u << left) - 1u;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) { s_pre[warp] = sum; s_cnt[warp] = __popc(m); }
    __syncthreads();
    int base = 0, total = 0;
#pragma unroll
    for (int w = 0; w < 8; w++) { base += s_pre[w] + (w < warp ? s_cnt[w] : 0); total += s_pre[w] + s_cnt[w]; }
    if (blockIdx.x == gridDim.x - 1 && blockIdx.y == 0 && tid == 0) *p.count = total;
    if (blockIdx.x == gridDim.x - 1 && !p.exact && p.T > AXPY_TC_TOKENS) {      // zeros behind the last position (k_axpy_tc reads stages of 64)
        const int64_t end = (total + 63) / 64 * 64 < p.coef_stride ? (total + 63) / 64 * 64 : p.coef_stride;
        for (int e = tid; e < UN * 64; e += 256)
            if (t0 + e / 64 < p.T && total + e % 64 < end) reinterpret_cast<__half *>(p.coef)[(size_t)(t0 + e / 64) * p.coef_stride + total + e % 64] = __ushort_as_half((unsigned short)0);
    }
    if (m == 0u) return;
    const int pos = base + __popc(m & ((1u << lane) - 1u));
    const bool mine = m >> lane & 1u;
    if (mine && blockIdx.y == 0) p.list[pos] = r;
    float o[UN];                                                      // (tokens beyond T too: no branch keeps the eight chains apart)
#pragma unroll
    for (int u = 0; u < UN; u++) {
        const bool on = in && !(l[u] < p.threshold);                  // (a NaN logit counts as active)
        if (!Q4) { o[u] = on ? v[u] : 0.f; continue; }
        o[u] = on || BLOCKS ? v[u] : fill;                            // what the graph leaves at an inactive neuron
    }
    if (Q4 && whole) {
        // A token's maximum is one instruction, and its two divisions are one lane's (256 tokens, 28672 neurons: with five shuffles a token and
        // divisions in every lane 29 us, the schedulers issuing in 78 % of the cycles; here 22).
        float am = 0.f;
#pragma unroll
        for (int u = 0; u < UN; u++) {
            float a;
            asm volatile("redux.sync.max.abs.f32 %0, %1, 0xffffffff;" : "=f"(a) : "f"(o[u]));     // (NaN values do not count, as in fmaxf)
            if ((lane & 7) == u) am = a;
        }
        const float id = am != 0.0f ? 127.0f / am : 0.0f, scale = round_f16(am / 127.0f);
#pragma unroll
        for (int u = 0; u < UN; u++) {
            const float q = (float)__float2int_rn(o[u] * __shfl_sync(0xffffffffu, id, u)) * __shfl_sync(0xffffffffu, scale, u);
            o[u] = in && !(l[u] < p.threshold) ? q : 0.f;
        }
    } else if (Q4) {                                                  // a bucket that cuts blocks: every row looks its own up
#pragma unroll
        for (int u = 0; u < UN; u++) {
            float amax = fabsf(o[u]);
            for (int k = 0; k < 32 && in && t0 + u < p.T; k++) amax = fmaxf(amax, fabsf(p.h[(size_t)(t0 + u) * p.h_stride + (g & ~(int64_t)31) + k]));
            const float id = amax != 0.0f ? 127.0f / amax : 0.0f;
            const float q = (float)__float2int_rn(o[u] * id) * round_f16(amax / 127.0f);
            o[u] = in && !(l[u] < p.threshold) ? q : 0.f;
        }
    }
    if (!mine) return;
#pragma unroll
    for (int u = 0; u < UN; u++) {
        if (t0 + u >= p.T) break;
        if (Q4 && p.exact) reinterpret_cast<float *>(p.coef)[(size_t)(t0 + u) * p.coef_stride + pos] = o[u];
        else reinterpret_cast<__half *>(p.coef)[(size_t)(t0 + u) * p.coef_stride + pos] = __float2half_rn(o[u]);
    }
}

int launch_coef(const CoefArgs & a, cudaStream_t st) {
    CoefP p;
    p.h = a.h; p.h_stride = a.h_stride; p.idx = a.idx; p.idx_stride = a.idx_stride; p.threshold = a.threshold;
    p.bucket = a.bucket; p.masks = a.masks; p.list = a.list_out; p.count = a.count_out; p.n_local = (int)a.n_local; p.T = a.T;
    p.fill_bias = a.fill_bias; p.coef = a.coef; p.coef_stride = a.coef_stride; p.exact = a.exact ? 1 : 0;
    const int n_chunks = (int)((a.n_local + 31) / 32);
    const dim3 grid((n_chunks + 7) / 8, (a.T + 7) / 8);
    if (a.wtype != PI_TYPE_Q4_0) PI_CUDA(launch_k(k_coef<false, false>, grid, dim3(256), 0, st, a.pdl, p));
    else if (a.h_uncleared)      PI_CUDA(launch_k(k_coef<true, false>, grid, dim3(256), 0, st, a.pdl, p));
    else                         PI_CUDA(launch_k(k_coef<true, true>, grid, dim3(256), 0, st, a.pdl, p));
    return PI_OK;
}

// ---------------------------------------------------------------------------------------------- launch
// At most 16 CTAs per slice (a partial vector each): more would cost the reader of the pieces more than they save.
// Tokens of a group: 8, 16, 32, or the equal share of up to 64 rounded up.  Few large groups expand a row's fragments less often, a group's
// products are made for all of its columns.  us with the groups taken | the others, 11008 x 4096 FP16 and 28672 x 8192 Q4_0 (exact):
//    40 tokens  1 x 40   43.2 |  1 x 48 44.4,   1 x 64  50.0,  2 x 32  48.6       233.6 |  272.7,  356.9,  371.3
//    80         2 x 40   64.5 |  2 x 48 67.2,   2 x 64  78.2,  3 x 32  71.1       448.1 |  525.7,  690.2,  557.4
//    96         2 x 48   71.9 |  3 x 40 82.0,   2 x 64  82.8,  3 x 32  74.1       536.3 |  652.5,  699.6,  565.9
//   128         2 x 64   93.6 |  4 x 40 103.3,  3 x 48  95.5,  4 x 32  95.4       715.6 |  863.0,  783.4,  748.7
//   256         4 x 64  163.6 |  7 x 40 168.5,  6 x 48 166.5,  8 x 32 172.4      1393.1 | 1504.3, 1545.9, 1478.7
static int axpy_mm_group(int T) {
    if (T <= 32) return T <= 8 ? 8 : T <= 16 ? 16 : 32;
    const int n = (T + 63) / 64, share = (T + n - 1) / n;
    return share <= 40 ? 40 : share <= 48 ? 48 : 64;
}

static void axpy_mm_shape(int64_t ncols, int T, int * n_cs, int * n_tg, int * grid, int * n_pieces) {
    const int group = axpy_mm_group(T);
    *n_cs = (int)((ncols + AX_CW - 1) / AX_CW);
    *n_tg = (T + group - 1) / group;
    const int n = *n_cs * *n_tg;
    *grid = (int)imin64(sm_count(), (int64_t)n * 16);
    *n_pieces = (*grid + n - 1) / n + 1;                              // ranges are not aligned to slices: one more than the quotient
}

// Which Q4_0 batches keep the CPU path's FP32 factors.  This is a promise about precision, not a matter of what the kernel can do: steps
// of 2..32 tokens over matrices of whole 1024 columns and at most 2^28 weights round weight and coefficient to FP16, everything else
// is exact.  Rounding buys (exact -> rounded) three layers of 28672 x 8192 and 8 tokens 576 -> 541 us per pass, a layer of 13824 x 5120
// and 16 tokens 85.9 -> 73.7 us.  A prompt keeps the factors that steps of the engine's batch have: exact where it takes one sequence.
bool axpy_mm_exact(int wtype, int64_t nrows, int64_t ncols, int T) {
    return wtype == PI_TYPE_Q4_0 && (T < 2 || T > 32 || ncols % 1024 != 0 || nrows * ncols > (int64_t)1 << 28);
}

int axpy_mm_least_pieces(int64_t ncols, int T) { int cs, tg, g, np; axpy_mm_shape(ncols, T, &cs, &tg, &g, &np); return np; }
int axpy_mm_pieces(int64_t ncols, int T) {
    const int least = axpy_mm_least_pieces(ncols, T), tc = T > AXPY_TC_TOKENS ? axpy_tc_pieces(ncols) : 0;
    return tc > least ? tc : least;
}

template <int MODE, int NT>
static int axpy_mm_go(const AxpyMmP & p, int grid, bool pdl, cudaStream_t st) {
    using Z = AxShape<MODE, NT>;
    static bool attr_done[16] = {false};
    int dev = 0;
    PI_CUDA(cudaGetDevice(&dev));
    auto kern = k_axpy_mm<MODE, NT>;
    const int smem = Z::HEAD + Z::S * Z::STAGE;
    if (dev >= 0 && dev < 16 && !attr_done[dev]) {
        PI_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        attr_done[dev] = true;
    }
    PI_CUDA(launch_k(kern, dim3(grid), dim3(AX_THREADS), (size_t)smem, st, pdl, p));
    return PI_OK;
}

template <int MODE>
static int axpy_mm_tokens(const AxpyMmP & p, int grid, bool pdl, cudaStream_t st) {
    switch (axpy_mm_group(p.T)) {
        case 8:  return axpy_mm_go<MODE, 1>(p, grid, pdl, st);
        case 16: return axpy_mm_go<MODE, 2>(p, grid, pdl, st);
        case 32: return axpy_mm_go<MODE, 4>(p, grid, pdl, st);
        case 40: return axpy_mm_go<MODE, 5>(p, grid, pdl, st);
        case 48: return axpy_mm_go<MODE, 6>(p, grid, pdl, st);
        default: return axpy_mm_go<MODE, 8>(p, grid, pdl, st);
    }
}

// PI_ERR_UNSUPPORTED: shape not eligible, the caller uses the CUDA-core kernel.
int launch_axpy_mm(const AxpyArgs & a, cudaStream_t st, int * pieces_used) {
    const bool q4 = a.wtype == PI_TYPE_Q4_0;
    if (!a.coef || a.coef_stride % 8 != 0 || !a.list || (q4 ? a.ncols % 256 != 0 : a.ncols % 8 != 0)) return PI_ERR_UNSUPPORTED;
    // (room for fewer partial vectors, an engine in a workspace of its earlier size: fewer and longer chains in tensor memory than here)
    if (a.T > AXPY_TC_TOKENS && !(q4 && a.exact) && a.n_groups >= axpy_tc_pieces(a.ncols)) return launch_axpy_tc(a, st, pieces_used);
    AxpyMmP p;
    int grid;
    axpy_mm_shape(a.ncols, a.T, &p.n_cs, &p.n_tg, &grid, &p.n_pieces);
    if (p.n_pieces > a.n_groups) return PI_ERR_UNSUPPORTED;
    p.Wt = (const uint8_t *)a.Wt; p.row_bytes = (int64_t)pi_row_bytes(a.wtype, a.ncols); p.nrows = (int)a.nrows; p.ncols = (int)a.ncols;
    p.nb = (int)(a.ncols / 32); p.T = a.T; p.list = a.list; p.count = a.count; p.coef = a.coef; p.coef_stride = a.coef_stride; p.partial = a.partial; p.status = a.status;
    if (pieces_used) *pieces_used = p.n_pieces;
    return q4 && a.exact ? axpy_mm_tokens<AX_Q4_EXACT>(p, grid, a.pdl, st) : q4 ? axpy_mm_tokens<AX_Q4>(p, grid, a.pdl, st) : axpy_mm_tokens<AX_F16>(p, grid, a.pdl, st);
}

}  // namespace pi
