// Mat-mat over planar Q4_0 rows for MORE than 32 tokens (prompt chunks of up to 256): the same operators, row selection and results as
// pi_mm.cu (masks and coefficients are FP16 rows' alone), another split of the work.  (FP16 rows: pi_mm_tc.cu.)
//
// Bound: the scaling of the Q4_0 blocks.  An mma of 16 rows x 32 columns x 8 tokens takes 8 clocks of a scheduler, the eight fused
// multiply-adds that apply its scales another 8 (as four packed ones they were slower, 259 us where these take 208: packed operations
// have half the pipes, and every row scale needed a copy).  What must not cost extra is shared memory: every warp reads its own
// fragments of both operands.
//
// Work split: as in pi_mm.cu every CTA takes an equal contiguous range of rows, in tiles of 192 (96), and producer warps (4) copy for the
// consumers (12) (a computing warp that issues cp.async waits while the SM's queue of outstanding loads is full: 700 to 2900 of the
// clocks of a stage).  Here all consumers share a stage (128 columns: 128 bytes of every activation, 64 of every row) and split the TILE:
// no partial sums, so the accumulators of a tile exist once and the tile can be 96 x 256.  Up to 128 tokens 6 x 2 consumers, beyond that 3 x 4,
// of 2 x 16 rows, the second of which a tile of up to half its height goes without; the token count of a consumer is a template argument in steps of 8 or 16, because a branch
// around every pair of products costs more than the products that it leaves out.
// Copies: the activations and dense rows come as TMA tiles (one instruction of one thread; with 16-byte cp.async the producers' own
// instruction rate, 50 clocks per warp and copy, bound every launch of few rows), gathered rows and the rows' scales by cp.async.
// The accumulators go straight to global memory: the ring runs on across tiles.
// Every wait is bounded, as in pi_mm.cu.
#include "pi_tc.cuh"

#include <type_traits>

namespace pi {

static constexpr int MW_THREADS = 512, MW_CONS = 12, MW_PROD = 128;       // warps 0 .. 11 consume, threads 384 .. 511 produce
static constexpr int MW_MT = 2;                         // fragments of 16 rows of a consumer
static constexpr int MW_SMEM_MAX = 224 * 1024;          // (leaves room for the static variables)
static constexpr int MW_SMAX = 6;                       // stages at most
static constexpr int MW_TOKENS = 256;                   // of a launch

struct alignas(64) MwP {
    CUtensorMap m_w, m_x, m_x2, m_d;                    // dense rows; activation: its low and high planes, its scales
    int per_tile;                                       // dense: rows of a tile
    const uint8_t * W; const uint8_t * W2; int64_t row_bytes; int nrows, ncols, nb;
    Act x; int T;
    const uint32_t * masks; const int32_t * bucket; int32_t * list; int32_t * count; unsigned long long * rows_total;
    const float * idx; int64_t idx_stride; float threshold;
    const float * bias; int relu;
    float * dst; __half * dst16; int64_t dst_stride;
    unsigned int * status;
    int n_slices, S;                                    // column slices of a row; stages
};

__device__ __forceinline__ void mw_cp16(uint32_t dst, const void * src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void mw_cp8(uint32_t dst, const void * src)  { asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" :: "r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void mw_arrive_copies(uint64_t * bar) { asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" :: "r"(smem_u32(bar)) : "memory"); }
__device__ __forceinline__ void mw_ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// (the C operand: four registers of their own, kept: as one value four times over it was copied into place for every product)
__device__ __forceinline__ void mw_imma(uint32_t (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const uint32_t (&c)[4]) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
}
// acc += (v - magic) * dd * d4: exact up to the two roundings of the products (see pi_mm.cu)
__device__ __forceinline__ void mw_scale_add(float & acc, uint32_t v, float dd, float md, float d4) { acc = fmaf(fmaf(__uint_as_float(v), dd, md), d4, acc); }

// WM x WN consumers of MT x 16 rows and NT x 8 tokens
template <int WM, int WN, int NT>
struct MwShape {
    static constexpr int TM = WM * MW_MT * 16, TN = WN * NT * 8;       // rows and tokens of a tile
    // 384 consumers + 128 producers share the 512 x 128 registers of the launch; producers of 192 gathered rows keep 12 addresses each
    static constexpr int REGS_C = WM == 6 ? 152 : 160, REGS_P = WM == 6 ? 56 : 32;
    static constexpr int KS = 128, WB = 64;                           // columns of a stage, bytes of a row's nibbles in it
    // a stage: rows [TM][64], activations' low plane [TN][64] and high plane [TN][64], rows' scales [TM][4 halves], activation
    // scales [TN][4 floats].  TMA writes and ldmatrix reads with the 16-byte pieces of a
    // row permuted by the row's number in groups of 8 (64-byte rows: pairs of rows in groups of 4), counted from 1024-byte boundaries.
    static constexpr int X_OFF = TM * WB, S_OFF = X_OFF + TN * 128, D_OFF = S_OFF + TM * 8, STAGE = (D_OFF + TN * 16 + 1023) / 1024 * 1024;
    static_assert(WM * WN == MW_CONS && X_OFF % 1024 == 0 && D_OFF % 128 == 0 && TN % 8 == 0 && TN <= 256, "split");
};

template <int WM, int WN, int NT, bool SPARSE, bool GATED>
__global__ void __launch_bounds__(MW_THREADS, 1) k_mm_wide(const __grid_constant__ MwP p) {
    using Z = MwShape<WM, WN, NT>;
    constexpr int TM = Z::TM, WB = Z::WB, MT = MW_MT;
    const int IT = GATED ? TM / 2 : SPARSE ? TM : p.per_tile;         // items (rows / neurons) of a tile
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char * smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    __shared__ int s_warp[MW_THREADS / 32];
    __shared__ uint64_t s_full[MW_SMAX], s_empty[MW_SMAX];
    __shared__ volatile int s_dead;
    int * rows = reinterpret_cast<int *>(smem + (size_t)p.S * Z::STAGE);          // rows of this CTA (sparse only)
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);    // (a shuffle: uniform for the compiler too; a branch it takes for divergent costs every mma behind it)
    const int wm = warp % WM, wn = warp / WM;
    const int G = gridDim.x, cta = blockIdx.x, S = p.S;
    const uint32_t ring = smem_u32(smem);
    constexpr uint32_t x_off = Z::X_OFF, s_off = Z::S_OFF, d_off = Z::D_OFF;
    if (tid < MW_SMAX) { mbar_init(s_full + tid, MW_PROD + 1); mbar_init(s_empty + tid, MW_CONS); }
    if (tid == 0) s_dead = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncthreads();
    pdl_launch();
    auto wait = [&](uint64_t * bar, unsigned parity) -> bool {        // warp-uniform; false: the wait ran out, here or elsewhere
        bool ok = false;
        for (int spins = 0; spins < (1 << 20) && !ok && !s_dead; spins++) ok = mbar_try_wait(bar, parity);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok && lane == 0) { s_dead = 1; if (p.status) atomicOr(p.status, 16u); }
        return ok;
    };

    int lo = 0, hi = 0, n_units = 0;
    auto set_range = [&](int n) {
        lo = (int)((long long)n * cta / G);
        hi = (int)((long long)n * (cta + 1) / G);
        n_units = (hi - lo + IT - 1) / IT * p.n_slices;
    };
    // ---- copies: a thread's pieces of a stage lie in the same rows for a whole tile
    constexpr int CW = WB / 16;                                       // 16-byte pieces of a row
    constexpr int NW = (TM * CW + MW_PROD - 1) / MW_PROD, WS = MW_PROD / CW;     // pieces of a thread, rows between them
    const int pt = tid - MW_CONS * 32;                              // producer thread
    const int cw = pt % CW;
    const uint8_t * wp[NW]; const uint8_t * sp[2] = {nullptr, nullptr};   // my pieces of the next slice; scales of rows pt, pt + 128
    unsigned w_ok = 0u;                                               // which of these rows exist
    int i_tile = 0, i_slice = 0;                                      // the unit that is requested next
    auto row_ptr = [&](int r, bool & ok) -> const uint8_t * {         // fragment row r of the tile (gated: 8 up rows, then their 8 gate rows)
        const int k = i_tile * IT + (GATED ? (r >> 4) * 8 + (r & 7) : r);
        ok = r < TM && lo + k < hi;
        return (GATED && (r & 8) ? p.W2 : p.W) + (ok ? (size_t)(SPARSE ? rows[k] : lo + k) * p.row_bytes : 0);
    };
    const int wr = pt / CW;
    const uint32_t w_to = (uint32_t)(wr * WB + ((cw ^ (wr >> 1)) & 3) * 16);
    auto issue_w = [&](int slot) {                                    // cp.async: addresses are kept and moved along
        if (i_slice == 0) {
            w_ok = 0u;
#pragma unroll
            for (int j = 0; j < (SPARSE ? NW : 0); j++) {
                bool ok;
                wp[j] = row_ptr(wr + j * WS, ok) + cw * 16;
                if (ok) w_ok |= 1u << j;
            }
#pragma unroll
            for (int j = 0; j < 2; j++) {
                bool ok;
                sp[j] = row_ptr(pt + j * MW_PROD, ok) + (size_t)p.nb * 16;
                if (ok) w_ok |= 1u << (NW + j);
            }
        }
        const uint32_t base = ring + (uint32_t)(slot * Z::STAGE);
#pragma unroll
        for (int j = 0; j < (SPARSE ? NW : 0); j++) {
            const uint32_t to = base + w_to + j * WS * WB;
            if (w_ok >> j & 1u) mw_cp16(to, wp[j]);
            wp[j] += WB;
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {
            if (w_ok >> (NW + j) & 1u) mw_cp8(base + s_off + (pt + j * MW_PROD) * 8, sp[j]);
            sp[j] += 8;
        }
    };
    auto issue_tma = [&](int slot) {                                  // one thread
        unsigned char * base = smem + (size_t)slot * Z::STAGE;
        uint64_t * bar = s_full + slot;
        mbar_expect_tx(bar, (unsigned)(Z::TN * 128 + Z::TN * 16 + (SPARSE ? 0 : p.per_tile * WB)));
        if (!SPARSE) tma_tile(smem_u32(base), &p.m_w, i_slice * 64, lo + i_tile * IT, bar);
        tma_tile(smem_u32(base + x_off), &p.m_x, i_slice * 64, 0, bar);
        tma_tile(smem_u32(base + x_off + Z::TN * 64), &p.m_x2, i_slice * 64, 0, bar);
        tma_tile(smem_u32(base + d_off), &p.m_d, i_slice * 4, 0, bar);
    };
    auto advance = [&]() { if (++i_slice == p.n_slices) { i_slice = 0; i_tile++; } };

    if (!SPARSE) {
        set_range(p.nrows);
        pdl_wait();                                                   // (the stages are many and long: nothing to gain before the wait)
    } else {
        pdl_wait();
        // ---- ranks of the active rows: thread t counts the words [c0, c1), a block scan gives the rank of its first row
        constexpr int KEEP = 4;
        const int n_chunks = (p.nrows + 31) / 32, per = (n_chunks + MW_THREADS - 1) / MW_THREADS;
        const int c0 = min(tid * per, n_chunks), c1 = min(c0 + per, n_chunks);
        auto word = [&](int c) {
            const uint32_t m = __ldcg(p.masks + c);
            const int left = p.nrows - c * 32;                        // bits beyond the last row never count
            return left < 32 ? m & ((1u << left) - 1u) : m;
        };
        uint32_t mw[KEEP];
        int mine = 0;
#pragma unroll
        for (int k = 0; k < KEEP; k++) { mw[k] = c0 + k < c1 ? word(c0 + k) : 0u; mine += __popc(mw[k]); }
        for (int c = c0 + KEEP; c < c1; c++) mine += __popc(word(c));
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        int before = 0, total = 0;
#pragma unroll
        for (int w = 0; w < MW_THREADS / 32; w++) { if (w < warp) before += s_warp[w]; total += s_warp[w]; }
        set_range(__shfl_sync(0xffffffffu, total, 0));
        if (cta == 0 && tid == 0) {
            if (p.count) *p.count = total;
            if (p.rows_total && total) atomicAdd(p.rows_total, (unsigned long long)total);      // statistics
        }
        int rank = before + incl - mine;
        for (int c = c0; c < c1 && rank < hi; c++) {
            uint32_t m = c - c0 < KEEP ? mw[0] : word(c);
            if (c - c0 < KEEP) {
#pragma unroll
                for (int k = 1; k < KEEP; k++) if (c - c0 == k) m = mw[k];
            }
            const int n = __popc(m);
            if (rank + n > lo) {
                for (int k = rank; m; k++) {
                    const int bit = __ffs(m) - 1;
                    m &= m - 1;
                    if (k >= lo && k < hi) rows[k - lo] = c * 32 + bit;
                }
            }
            rank += n;
        }
        __syncthreads();
        if (p.list) for (int k = tid; k < hi - lo; k += MW_THREADS) p.list[lo + k] = rows[k];
    }
    if (warp >= MW_CONS) {
        // ================================================================= producers
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" :: "n"(Z::REGS_P));
        int slot = 0;
        unsigned phase = 1u;                                          // parity of the hand-back to wait for (first round: none)
        int i = 0;
        for (; i < n_units; i++) {
            if (!wait(s_empty + slot, phase)) break;
            if (pt == 0) issue_tma(slot);
            issue_w(slot);
            mw_arrive_copies(s_full + slot);
            advance();
            if (++slot == S) { slot = 0; phase ^= 1u; }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (pt == 0) ring_land(s_full, i, S);
        return;
    }
    // ===================================================================== consumers
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" :: "n"(Z::REGS_C));
    float acc[MT][NT][4];
    auto clear = [&]() {
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
            for (int n = 0; n < NT; n++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[m][n][j] = 0.f;
    };
    clear();
    const int g = lane >> 2, q = lane & 3;
    uint32_t MAGIC[4];
#pragma unroll
    for (int j = 0; j < 4; j++) asm volatile("mov.u32 %0, 0x4B400000;" : "=r"(MAGIC[j]));
    // This warp's part of the tile: 16 rows from row0 and 16 from row0 + MS.  6 consumers along the rows: the second fragments lie above all
    // first ones, and a tile of up to 96 rows has none (104 gathered rows are one tile instead of a whole one and a nearly empty one).
    // 3 consumers: neighbours, so that 56 rows are two consumers' work and not three's; always multiplied.
    constexpr bool APART = WM == 6;
    constexpr int MS = APART ? WM * 16 : 16;
    const int row0 = wm * (APART ? 16 : 32), tok0 = wn * NT * 8;
    // ldmatrix row addresses inside a stage (fragment layouts of mma.m16n8k16 / m16n8k32); the piece is added per step
    const uint32_t a_row = (uint32_t)((row0 + (lane & 15) + (lane >> 4) * MS) * WB);
    constexpr int XB = 64;                                            // bytes of a token in a plane
    const uint32_t plane = ((lane >> 3) & 1) * Z::TN * 64;
    const uint32_t b_row = x_off + plane + (uint32_t)((tok0 + (lane & 7) + (lane >> 4) * 8) * XB), b_last = x_off + plane + (uint32_t)((tok0 + (NT - 1) * 8 + (lane & 7)) * XB);
    const int a_swz = (lane >> 1) & 3, b_swz = (lane & 7) >> 1;

    int tile = 0, slice = 0, slot = 0;
    unsigned phase = 0u;
    for (int i = 0; i < n_units; i++) {
        if (!wait(s_full + slot, phase)) break;
        const uint32_t base = ring + (uint32_t)(slot * Z::STAGE);
        const int n_tile = min(IT, hi - lo - tile * IT);              // items
        const bool busy = (GATED ? row0 / 2 : row0) < n_tile && tok0 < p.T;       // my rows and tokens exist
        auto multiply = [&](auto mc) {                                // MC fragments of 16 rows
            constexpr int MC = decltype(mc)::value;
#pragma unroll
            for (int k = 0; k < 4; k++) {                         // block by block
                uint32_t w[4], a[MC][4];
                mw_ldsm4(w, base + a_row + ((k ^ a_swz) & 3) * 16);
                float d4[MC][2];                                  // (the nibbles stand for 16 times their value)
#pragma unroll
                for (int m = 0; m < MC; m++) {
                    const uint32_t w0 = w[2 * m], wh = w[2 * m + 1];
                    a[m][0] = ((w0 << 4) & 0xF0F0F0F0u) ^ 0x80808080u; a[m][1] = ((wh << 4) & 0xF0F0F0F0u) ^ 0x80808080u;
                    a[m][2] = (w0 & 0xF0F0F0F0u) ^ 0x80808080u;        a[m][3] = (wh & 0xF0F0F0F0u) ^ 0x80808080u;
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        unsigned short s;
                        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(s) : "r"(base + s_off + (row0 + m * MS + g + h * 8) * 8 + k * 2));
                        d4[m][h] = __half2float(__ushort_as_half(s)) * 0.0625f;
                    }
                }
#pragma unroll
                for (int n = 0; n < NT; n += 2) {
                    uint32_t b[4];
                    mw_ldsm4(b, base + (n + 1 < NT ? b_row + n * 8 * XB : b_last) + ((k ^ b_swz) & 3) * 16);
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        if (n + u >= NT) break;
                        float t0, t1;                             // scales of tokens 2q, 2q + 1
                        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(t0) : "r"(base + d_off + (tok0 + (n + u) * 8 + 2 * q) * 16 + k * 4));
                        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(t1) : "r"(base + d_off + (tok0 + (n + u) * 8 + 2 * q + 1) * 16 + k * 4));
                        const float m0 = t0 * -12582912.0f, m1 = t1 * -12582912.0f;
#pragma unroll
                        for (int m = 0; m < MC; m++) {
                            uint32_t c[4];
                            mw_imma(c, a[m], b[2 * u], b[2 * u + 1], MAGIC);
                            float (&o)[4] = acc[m][(n + u) % NT];
                            mw_scale_add(o[0], c[0], t0, m0, d4[m][0]);
                            mw_scale_add(o[1], c[1], t1, m1, d4[m][0]);
                            mw_scale_add(o[2], c[2], t0, m0, d4[m][1]);
                            mw_scale_add(o[3], c[3], t1, m1, d4[m][1]);
                        }
                    }
                }
            }
        };
        if (!busy) {
        } else if (!APART || (GATED ? MS / 2 : MS) < n_tile) {
            multiply(std::integral_constant<int, 2>());
        } else {
            multiply(std::integral_constant<int, APART ? 1 : 2>());
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(s_empty + slot);                   // handed back
        if (++slot == S) { slot = 0; phase ^= 1u; }
        if (slice == p.n_slices - 1) {
            // ---- the tile is complete: a lane holds rows g and g + 8 of each fragment (gated: up and gate of one item), tokens 2q, 2q + 1
            if (busy) {
#pragma unroll
                for (int m = 0; m < MT; m++) {
#pragma unroll
                    for (int h = 0; h < (GATED ? 1 : 2); h++) {
                        const int k = GATED ? (row0 + m * MS) / 2 + g : row0 + m * MS + g + h * 8;     // item of the tile
                        if (k < n_tile) {
                            const int item = lo + tile * IT + k;
                            const int r = SPARSE ? rows[tile * IT + k] : item;
                            const int64_t gid = SPARSE && p.bucket ? p.bucket[r] : r;
                            const float bias = p.bias ? p.bias[gid] : 0.f;
#pragma unroll
                            for (int n = 0; n < NT; n++) {
#pragma unroll
                                for (int j = 0; j < 2; j++) {
                                    const int t = tok0 + n * 8 + 2 * q + j;
                                    if (t >= p.T) continue;
                                    const float v[2] = {acc[m][n][j], acc[m][n][2 + j]};
                                    float o = GATED ? fmaxf(v[1], 0.f) * v[0] : v[h];
                                    const bool off = SPARSE && p.idx[(size_t)t * p.idx_stride + gid] < p.threshold;   // (a NaN logit counts as active)
                                    if (off) o = 0.f;
                                    if (p.bias) o += bias;
                                    if (p.relu) o = fmaxf(o, 0.f);
                                    if (p.dst)   p.dst[(size_t)t * p.dst_stride + gid] = o;
                                    if (p.dst16) p.dst16[(size_t)t * p.dst_stride + gid] = __float2half_rn(o);
                                }
                            }
                        }
                    }
                }
            }
            __syncwarp();                                             // (keeps the compiler from folding what follows into the loop: 9000 x 4096, 128 tokens 65 us, so 50)
            clear();
        }
        if (++slice == p.n_slices) { slice = 0; tile++; }
    }
}

// ---------------------------------------------------------------------------------------------- launch
typedef CUresult (*MwEncode)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                             CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int tensor_map(CUtensorMap * m, CUtensorMapDataType type, const void * base, int64_t cols, int64_t rows, int64_t pitch, int box_cols, int box_rows, CUtensorMapSwizzle swizzle) {
    static MwEncode encode = nullptr;
    if (!encode) {
        void * f = nullptr;
        cudaDriverEntryPointQueryResult q;
        PI_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q));
        PI_REQUIRE(f && q == cudaDriverEntryPointSuccess, "mm_wide: the driver has no cuTensorMapEncodeTiled");
        encode = (MwEncode)f;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)pitch};
    const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows}, steps[2] = {1, 1};
    const CUresult rc = encode(m, type, 2, const_cast<void *>(base), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    PI_REQUIRE(rc == CUDA_SUCCESS, "mm_wide: tensor map refused (%d): %lld x %lld, pitch %lld", (int)rc, (long long)rows, (long long)cols, (long long)pitch);
    return PI_OK;
}

template <int WM, int WN, int NT, bool SPARSE, bool GATED>
static int mw_go(MwP p, bool pdl, cudaStream_t st) {
    using Z = MwShape<WM, WN, NT>;
    p.n_slices = (p.ncols + Z::KS - 1) / Z::KS;
    const int G = (int)imin64(sm_count(), (p.nrows + 7) / 8);
    const int list = SPARSE ? ((p.nrows + G - 1) / G + 1) * 4 : 0;    // bytes
    if (list > 8192) return PI_ERR_UNSUPPORTED;                       // (more than MM_MAX_ROWS rows)
    p.S = (MW_SMEM_MAX - 1024 - list) / Z::STAGE;
    if (p.S > MW_SMAX) p.S = MW_SMAX;
    static_assert(2 * Z::STAGE <= MW_SMEM_MAX - 1024 - 8192, "two stages");
    p.per_tile = 0;
    int rc;
    if (!SPARSE) {                                                    // equal tiles
        const int share = (p.nrows + G - 1) / G, tiles = (share + Z::TM - 1) / Z::TM;
        p.per_tile = (share + tiles - 1) / tiles;
        rc = tensor_map(&p.m_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, p.W, (int64_t)p.nb * 16, p.nrows, p.row_bytes, 64, p.per_tile, CU_TENSOR_MAP_SWIZZLE_64B);
        if (rc != PI_OK) return rc;
    }
    if ((rc = tensor_map(&p.m_x, CU_TENSOR_MAP_DATA_TYPE_UINT8, p.x.lo, (int64_t)p.nb * 16, p.T, (int64_t)p.nb * 16, 64, Z::TN, CU_TENSOR_MAP_SWIZZLE_64B)) != PI_OK) return rc;
    if ((rc = tensor_map(&p.m_x2, CU_TENSOR_MAP_DATA_TYPE_UINT8, p.x.hi, (int64_t)p.nb * 16, p.T, (int64_t)p.nb * 16, 64, Z::TN, CU_TENSOR_MAP_SWIZZLE_64B)) != PI_OK) return rc;
    if ((rc = tensor_map(&p.m_d, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, p.x.d, p.nb, p.T, (int64_t)p.nb * 4, 4, Z::TN, CU_TENSOR_MAP_SWIZZLE_NONE)) != PI_OK) return rc;
    static bool attr_done[16] = {false};
    int dev = 0;
    PI_CUDA(cudaGetDevice(&dev));
    auto kern = k_mm_wide<WM, WN, NT, SPARSE, GATED>;
    if (dev >= 0 && dev < 16 && !attr_done[dev]) {
        PI_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MW_SMEM_MAX));
        attr_done[dev] = true;
    }
    PI_CUDA(launch_k(kern, dim3(G), dim3(MW_THREADS), (size_t)p.S * Z::STAGE + list + 1024, st, pdl, p));
    return PI_OK;
}

template <int WM, int WN, int NT>
static int mw_sel(const MwP & p, bool pdl, cudaStream_t st) {
    if (!p.masks) return mw_go<WM, WN, NT, false, false>(p, pdl, st);
    if (p.W2)     return mw_go<WM, WN, NT, true, true>(p, pdl, st);
    return mw_go<WM, WN, NT, true, false>(p, pdl, st);
}

// The narrowest tile that holds the tokens: the products of a tile are made for all of its columns.  us at this step | at the next wider one,
// 10240 x 8192: 64 tokens 69.2 | 81.7; 80 82.8 | 96.0; 96 96.5 | 113.7; 128 114.6 | 144.1; 192 148.7 | 189.6.  (2..32 tokens go to k_mm.)  Steps at 112, 160 and 224 would give token
// counts below them up to half of those differences, for six more instances each.
static int mw_tokens(const MwP & p, bool pdl, cudaStream_t st) {
    if (p.T <= 64)  return mw_sel<6, 2, 4>(p, pdl, st);
    if (p.T <= 80)  return mw_sel<6, 2, 5>(p, pdl, st);
    if (p.T <= 96)  return mw_sel<6, 2, 6>(p, pdl, st);
    if (p.T <= 128) return mw_sel<6, 2, 8>(p, pdl, st);
    if (p.T <= 192) return mw_sel<3, 4, 6>(p, pdl, st);
    return mw_sel<3, 4, 8>(p, pdl, st);
}

// Called by launch_mm, which has checked the arguments.  Tokens go in launches of at most 256.
int launch_mm_wide(const GemvArgs & a, cudaStream_t st) {
    for (int t0 = 0; t0 < a.T; t0 += MW_TOKENS) {
        MwP p;
        p.W = (const uint8_t *)a.W; p.W2 = (const uint8_t *)a.W2; p.row_bytes = (int64_t)pi_row_bytes(a.wtype, a.ncols);
        p.nrows = (int)a.nrows; p.ncols = (int)a.ncols; p.nb = (int)(a.ncols / 32);
        p.T = a.T - t0 < MW_TOKENS ? a.T - t0 : MW_TOKENS;
        p.x.lo = a.x.lo + (size_t)t0 * p.nb; p.x.hi = a.x.hi + (size_t)t0 * p.nb; p.x.d = a.x.d + (size_t)t0 * p.nb;
        p.masks = a.masks; p.bucket = a.bucket; p.list = a.list_out; p.count = a.count_out; p.rows_total = t0 == 0 ? a.rows_total : nullptr;
        p.idx = a.idx ? a.idx + (size_t)t0 * a.idx_stride : nullptr; p.idx_stride = a.idx_stride; p.threshold = a.threshold;
        p.bias = a.bias; p.relu = a.relu;
        p.dst = a.dst ? a.dst + (size_t)t0 * a.dst_stride : nullptr;
        p.dst16 = a.dst16 ? a.dst16 + (size_t)t0 * a.dst_stride : nullptr; p.dst_stride = a.dst_stride;
        p.status = a.status;
        const int rc = mw_tokens(p, a.pdl, st);
        if (rc != PI_OK) return rc;
    }
    return PI_OK;
}

}  // namespace pi
