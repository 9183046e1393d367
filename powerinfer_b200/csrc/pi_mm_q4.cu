// Mat-mat over planar Q4_0 rows of many columns for MORE than 96 tokens (prompt chunks; the lines: mm_q4_takes) on tcgen05: the operators, row
// selection and results of pi_mm.cu (masks and coefficients are FP16 rows' alone).
//
// A term is (q - 8) * w * v * d: an integer and an FP16 scale of the row's block, an int8 and an FP16 scale of the token's block.  (q - 8) * w has 15
// significant bits, v * d 18, and both are multiples of 2^-24: each is exactly the sum of TWO halves, its rounding and the rest.  Of
// the four products of halves the two rests' (up to 2^-22 of the term, each rest up to 2^-11 of its value) is left out; the other three are exact
// in FP32.  So the scales ride on the operands and the tensor cores do all of the work; as integers per block, scaled one by one, 2.7e9 sums of 256
// tokens and a 70B-shape gather take two FP32 instructions each (mma.sync 770 us, here 530; tcgen05 kind::i8 with that scaling 600 .. 700).  The
// fourth product costs 4 .. 5 % (10240 x 8192, 256 tokens 128 -> 134 us) for 2 % of the error.
//
// Precision: the tensor cores cut FP32 sums at every step, so a sum must not stay with them.  After 64 columns
// it is drained and added with rounding in registers; the small products of a drain come first, so that only the four large
// ones cut anything.  A sum that fits FP32 at every step (whole numbers at scales that are powers of two) is exact.  Error against 64 bits, one FP32
// chain of all blocks (pi_mm_wide.cu) | here: random values in 8192 columns 2.86e-7 | 2.32e-7, 4096 2.03e-7 | 1.84e-7, 3072 1.77e-7 | 1.69e-7, 2816
// 1.69e-7 | 1.65e-7, 2560 1.61e-7 | 1.61e-7, 2048 1.44e-7 | 1.53e-7: shorter sums stay there (mm_q4_takes).  A token with one feature that is not zero
// 2.5e-8 | 5.5e-8 (what is left out, and a cut in the place of a rounding), with 16 6.8e-8 | 8.9e-8, with every 16th 2.6e-7 | 2.1e-7.  (A drain
// times 1 + 2^-23, what cutting four times takes on the average, would halve the bias of random sums, 2.18e-7 in 8192 columns, and move exact ones.)
// A row with a scale above 8188 may leave the halves' range, 65504: its sums are not finite then, and are made anew block by block.
//
// Tokens are the 128 lanes (M), rows the columns (N, steps of 16): every CTA takes its equal contiguous range of rows, in tiles of up to 160.
// More than 128 tokens: neighbouring CTAs take the same rows for other tokens (the second finds them in L2).
//
// Warps: 0 issues the products; 1 brings the activations' bytes as TMA tiles; 4..7 make the tokens' halves of them and store these to TENSOR
// memory, where the products read them (from shared memory both operands would take 174 of its 128 bytes per clock); 2, 3, 8..11 and
// 20..23 make the rows' halves in shared memory, 16 rows x 2 blocks a warp and stage; 12..19 drain, each 32 tokens x half of the rows.
// (A token is a lane from the tensor memory on: loading its bytes there straight from global memory touched 32 lines an instruction and took
// half of the load pipe's time.)
#include "pi_tc.cuh"

#include <type_traits>

namespace pi {

static constexpr int TS_THREADS = 768, TS_CONS = 8, TS_WARPS_W = 10;   // draining warps, warps that bring rows
static constexpr int TS_TOK = 128, TS_NC = 80, TS_N = 2 * TS_NC;      // tokens of a tile; columns of a draining group of four warps, of a tile
static constexpr int TS_REGS_S = 56, TS_REGS_X = 80, TS_REGS_C = 112; // 3 x 56 + 80 + 2 x 112 warpgroups' shares of the 6 x 80 of the launch
static constexpr int TS_SMAX = 10;                                    // stages of rows at most (no fewer than TS_WARPS_W: a warp that has every tenth
                                                                      // stage must not be two uses of a slot ahead of the products)
static constexpr int TS_EPI = 16 * 34 * 4;                            // a warp's transposition of 16 rows x 32 tokens
static constexpr int TS_SMEM_MAX = 226 * 1024;
static constexpr uint32_t TS_XBUF = 2 * TS_TOK * 64 + TS_TOK * 16;    // activations of 128 columns: low halves of four blocks, high halves, scales
static constexpr uint32_t TS_A = 2 * TS_N;                            // tensor memory: two buffers of sums, two of token halves (32 + 32 columns)

struct alignas(64) TsP {
    CUtensorMap m_lo, m_hi, m_d;
    const uint8_t * W; const uint8_t * W2; int64_t row_bytes; int nrows, nb;
    Act x; int T, n_tt, groups, ring;                                 // tiles of tokens; groups of CTAs along the rows; bytes of the ring
    const uint32_t * masks; const int32_t * bucket; int32_t * list; int32_t * count; unsigned long long * rows_total;
    const float * idx; int64_t idx_stride; float threshold;
    const float * bias; int relu;
    float * dst; __half * dst16; int64_t dst_stride;
    unsigned int * status;
};

__device__ __forceinline__ uint32_t ts_mul2(uint32_t a, uint32_t b) { uint32_t r; asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ uint32_t ts_add2(uint32_t a, uint32_t b) { uint32_t r; asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ uint32_t ts_fma2(uint32_t a, uint32_t b, uint32_t c) { uint32_t r; asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c)); return r; }
__device__ __forceinline__ uint32_t ts_neg2(uint32_t a) { uint32_t r; asm("neg.f16x2 %0, %1;" : "=r"(r) : "r"(a)); return r; }     // (folds into the next one)
// a * b = hi + lo, exactly
__device__ __forceinline__ void ts_split(uint32_t a, uint32_t b, uint32_t & hi, uint32_t & lo) { hi = ts_mul2(a, b); lo = ts_fma2(a, b, ts_neg2(hi)); }
// Token scales above 256 (products with 127 above the halves' range) are brought below by a power of two per token and block, which the
// drain takes back: its exponent.  A CTA with such a token drains every block by itself (one power for two blocks would make a subnormal
// half of the smaller scale, and lose what the row's result consists of where its weights in the larger one are 0).
__device__ __forceinline__ int ts_down(float d) { const int e = (int)(__float_as_uint(d) >> 23) - 127; return max(0, e - 7); }

// The rare rows whose scales times 8 are above the halves' range: found, and summed block by block for one token
__device__ __forceinline__ bool ts_beyond(unsigned short s) { return (s & 0x7FFFu) > 0x6FFFu; }      // |s| > 8188, infinite or NaN
__device__ __forceinline__ bool ts_row_beyond(const uint8_t * row, int nb, int lane) {               // (the same row in all lanes)
    const unsigned short * s = reinterpret_cast<const unsigned short *>(row + (size_t)nb * 16);
    bool any = false;
    for (int b = lane; b < nb; b += 32) any |= ts_beyond(s[b]);
    return __any_sync(0xffffffffu, any);
}
__device__ __forceinline__ float ts_row_sum(const uint8_t * row, const uint4 * lo, const uint4 * hi, const float * d, int nb) {
    const unsigned short * s = reinterpret_cast<const unsigned short *>(row + (size_t)nb * 16);
    float acc = 0.f;
#pragma unroll 1
    for (int b = 0; b < nb; b++) {
        const uint4 q = reinterpret_cast<const uint4 *>(row)[b], l = lo[b], h = hi[b];
        const uint32_t qs[4] = {q.x, q.y, q.z, q.w}, ls[4] = {l.x, l.y, l.z, l.w}, hs[4] = {h.x, h.y, h.z, h.w};
        int sum = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {                                 // (q - 8: nibbles as signed bytes)
            sum = __dp4a((int)__vsub4(qs[j] & 0x0F0F0F0Fu, 0x08080808u), (int)ls[j], sum);
            sum = __dp4a((int)__vsub4(qs[j] >> 4 & 0x0F0F0F0Fu, 0x08080808u), (int)hs[j], sum);
        }
        acc = fmaf((float)sum, __half2float(__ushort_as_half(s[b])) * d[b], acc);
    }
    return acc;
}

template <bool SPARSE, bool GATED>
__global__ void __launch_bounds__(TS_THREADS, 1) k_mm_q4(const __grid_constant__ TsP p) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ int s_warp[TS_THREADS / 32];
    __shared__ uint64_t s_full[TS_SMAX], s_empty[TS_SMAX], s_xfull[2], s_xempty[2], s_dfull[2], s_dempty[2], s_fin;
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_dead;
    __shared__ int s_large;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);    // (uniform for the compiler)
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t xbufs = ring + (uint32_t)p.ring;
    float * const epi = reinterpret_cast<float *>(smem_raw + (xbufs - smem_u32(smem_raw)) + 2 * TS_XBUF);
    int * const rows = reinterpret_cast<int *>(epi + TS_CONS * (TS_EPI / 4));      // rows of this CTA (sparse only)
    const int grp = blockIdx.x / p.n_tt, tok0 = (int)(blockIdx.x % p.n_tt) * TS_TOK;
    const int Tt = min(TS_TOK, p.T - tok0), live_quarters = (Tt + 31) / 32;        // tokens of this tile
    if (tid == 0) { s_dead = 0; s_large = 0; }
    if (warp == 0) tc_alloc(&s_tmem, 512);
    pdl_launch();
    pdl_wait();
    int lo, hi;
    if (SPARSE) {
        const int total = tc_active_rows<TS_THREADS>(p.masks, p.nrows, grp, p.groups, s_warp, rows, lo, hi);
        if (blockIdx.x == 0 && tid == 0) {
            if (p.count) *p.count = total;
            if (p.rows_total && total) atomicAdd(p.rows_total, (unsigned long long)total);      // statistics
        }
        if (p.list && tok0 == 0) for (int k = tid; k < hi - lo; k += TS_THREADS) p.list[lo + k] = rows[k];
    } else {
        lo = (int)((long long)p.nrows * grp / p.groups);
        hi = (int)((long long)p.nrows * (grp + 1) / p.groups);
    }
    // tiles of equal height (gated: column pairs, up and gate of one item)
    const int n_cols = (hi - lo) * (GATED ? 2 : 1), n_tiles = (n_cols + TS_N - 1) / TS_N;
    const int N = n_tiles ? ((n_cols + n_tiles - 1) / n_tiles + 15) / 16 * 16 : 16, nc = N / 2;
    const int items = GATED ? N / 2 : N;                              // of a tile
    const int n_st = p.nb / 2;                                        // stages of 64 columns: two blocks
    const uint32_t slot_bytes = (uint32_t)N * 256u;                   // rounded halves of all rows, then the rests
    const int S = min(TS_SMAX, p.ring / (int)slot_bytes);
    const int tasks = N / 16;                                         // of a stage of rows
    if (tid < TS_SMAX) { mbar_init(s_full + tid, (unsigned)(tasks + live_quarters)); mbar_init(s_empty + tid, 1); }
    if (tid < 2) { mbar_init(s_dfull + tid, 1); mbar_init(s_dempty + tid, (unsigned)live_quarters * 2); }
    if (tid < 2) { mbar_init(s_xfull + tid, 1); mbar_init(s_xempty + tid, (unsigned)live_quarters); }
    if (tid == 0) mbar_init(&s_fin, 1);
    if (n_tiles) {                                                    // a scale above 256? (ts_down; NaN too)
        bool large = false;
        const float4 * d4 = reinterpret_cast<const float4 *>(p.x.d + (size_t)tok0 * p.nb);
        for (int e = tid; e < Tt * p.nb / 4; e += TS_THREADS) { const float4 v = d4[e]; large |= !(fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)) <= 256.f); }
        if (__any_sync(0xffffffffu, large) && lane == 0) atomicOr(&s_large, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem, 0);
    const bool large = __shfl_sync(0xffffffffu, s_large, 0);
    auto wait = [&](uint64_t * bar, unsigned parity) -> bool {        // warp-uniform; false: the wait ran out, here or elsewhere
        bool ok = __all_sync(0xffffffffu, mbar_try_wait(bar, parity));
        if (__builtin_expect(ok, 1)) return true;
        for (int spins = 0; spins < (1 << 20) && !ok && !s_dead; spins++) ok = mbar_try_wait(bar, parity);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok && lane == 0) { s_dead = 1; if (p.status) atomicOr(p.status, 16u); }
        return ok;
    };

    if (warp < 4 || (warp >= 8 && warp < 12) || warp >= 20) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" :: "n"(TS_REGS_S));
        if (warp == 0) {
            // ============================================================= products
            const uint32_t idesc = tc_idesc(N, false);
            int slot = 0, ab = 0, db = 0;
            unsigned phase = 0u, dphase = 1u;                         // (the first round's buffers of sums are free)
            for (int i = 0; i < n_tiles * n_st; i++) {
                if (!wait(s_full + slot, phase)) break;               // rows and tokens (one barrier: a wait that is over costs 150 clocks)
                const uint32_t a = tmem + TS_A + (uint32_t)ab * 64u;
                const uint64_t w = tc_desc_k(ring + (uint32_t)slot * slot_bytes), w_rest = tc_desc_k(ring + (uint32_t)slot * slot_bytes + (uint32_t)N * 128u);
                auto drained = [&](auto first, auto last) {           // products of columns 16 first .. 16 last
                    constexpr int K0 = decltype(first)::value, K1 = decltype(last)::value;
                    wait(s_dempty + db, dphase);
                    tc_fence_after();
                    const uint32_t d = tmem + (uint32_t)db * TS_N;
#pragma unroll
                    for (int k = K0; k < K1; k++) {                   // the rests first (see above)
                        tc_mma_f16_ta(d, a + 32u + 8u * k, w + 2 * k, idesc, k > K0);
                        tc_mma_f16_ta(d, a + 8u * k, w_rest + 2 * k, idesc, true);
                    }
#pragma unroll
                    for (int k = K0; k < K1; k++) tc_mma_f16_ta(d, a + 8u * k, w + 2 * k, idesc, true);
                    tc_commit(s_dfull + db);
                    db ^= 1;
                    if (db == 0) dphase ^= 1u;
                };
                if (!large) drained(std::integral_constant<int, 0>(), std::integral_constant<int, 4>());
                else {
                    drained(std::integral_constant<int, 0>(), std::integral_constant<int, 2>());
                    drained(std::integral_constant<int, 2>(), std::integral_constant<int, 4>());
                }
                tc_commit(s_empty + slot);
                if (++slot == S) { slot = 0; phase ^= 1u; }
                ab ^= 1;
            }
            tc_commit(&s_fin);                                        // nothing is in flight when tensor memory is given back
            for (int spins = 0; spins < (1 << 20) && !mbar_try_wait(&s_fin, 0u); spins++) {}
            __syncwarp();
        } else if (warp == 1) {
            // ============================================================= activations
            int xb = 0, pair = 0;
            unsigned xphase = 1u;
            int i = 0;
            for (; i < n_tiles * (n_st / 2); i++) {
                if (!wait(s_xempty + xb, xphase)) break;
                if (lane == 0) {
                    const uint32_t to = xbufs + (uint32_t)xb * TS_XBUF;
                    mbar_expect_tx(s_xfull + xb, TS_XBUF);
                    tma_tile(to, &p.m_lo, pair * 64, tok0, s_xfull + xb);
                    tma_tile(to + TS_TOK * 64, &p.m_hi, pair * 64, tok0, s_xfull + xb);
                    tma_tile(to + 2 * TS_TOK * 64, &p.m_d, pair * 4, tok0, s_xfull + xb);
                }
                __syncwarp();
                if (++pair == n_st / 2) pair = 0;
                xb ^= 1;
                if (xb == 0) xphase ^= 1u;
            }
            if (lane == 0) ring_land(s_xfull, i, 2);
            __syncwarp();
        } else {
            // ============================================================= rows: a block a lane, 16 rows x 2 blocks
            // A warp has the same 16 rows of a tile in every `turns`-th stage: its addresses only move along (looking its next 16 rows up each time
            // took a third of its time).
            const int pw = warp < 4 ? warp - 2 : warp < 12 ? warp - 6 : warp - 14, turns = TS_WARPS_W / tasks, part = pw % tasks;
            if (pw < tasks * turns && n_tiles) {
                const int r = part * 16 + (lane & 15), blk = lane >> 4, n_all = n_tiles * n_st;
                const uint8_t * src, * scale;
                int l_i = pw / tasks, l_st = l_i, l_tile = 0;         // the stage that is requested next, of all and of the tile
                while (l_st >= n_st) { l_st -= n_st; l_tile++; }
                auto rows_of = [&](int tile) {
                    const int item = min(tile * items + (GATED ? r >> 1 : r), hi - lo - 1);       // (a column of no row: the last)
                    const size_t row = (size_t)(SPARSE ? rows[item] : lo + item);
                    const uint8_t * at = (GATED && (r & 1) ? p.W2 : p.W) + row * p.row_bytes;
                    src = at + (size_t)(l_st * 2 + blk) * 16;
                    scale = at + (size_t)p.nb * 16 + (size_t)(l_st * 2 + blk) * 2;
                };
                rows_of(l_tile);
                uint4 q[3];
                unsigned short sc[3];
                auto load = [&](uint4 & v, unsigned short & s) {
                    if (l_i >= n_all) return;
                    v = ldg_stream(src);
                    s = __ldg(reinterpret_cast<const unsigned short *>(scale));
                    src += turns * 32; scale += turns * 4;
                    l_i += turns; l_st += turns;
                    if (l_st >= n_st && l_i < n_all) {
                        while (l_st >= n_st) { l_st -= n_st; l_tile++; }
                        rows_of(l_tile);
                    }
                };
                int i = pw / tasks, slot = i;                         // the stage that is stored next (slots: no fewer than turns)
                unsigned phase = 1u;
                bool ok = true;
                const uint32_t mine = ring + (uint32_t)(r * 128);
                auto store = [&](const uint4 & v, unsigned short s) {
                    if (i >= n_all) return;
                    ok = wait(s_empty + slot, phase) && ok;
                    const uint32_t at = mine + (uint32_t)slot * slot_bytes, s2 = (uint32_t)s * 0x10001u, w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int j = 0; j < 4; j++) {                     // bytes 4j .. 4j + 3: columns {0, 2, 1, 3} and 16 + {0, 2, 1, 3} of them
                        uint32_t h[4], l[4];                          // (bit patterns: 0x6400 = 1024, 0x2C00 = 1/16, 0xE408 = -1032, 0xD480 = -72)
                        const uint32_t x = w[j], y = w[j] >> 8;
                        ts_split(ts_add2((x & 0x000F000Fu) | 0x64006400u, 0xE408E408u), s2, h[0], l[0]);
                        ts_split(ts_add2((y & 0x000F000Fu) | 0x64006400u, 0xE408E408u), s2, h[1], l[1]);
                        ts_split(ts_fma2((x & 0x00F000F0u) | 0x64006400u, 0x2C002C00u, 0xD480D480u), s2, h[2], l[2]);
                        ts_split(ts_fma2((y & 0x00F000F0u) | 0x64006400u, 0x2C002C00u, 0xD480D480u), s2, h[3], l[3]);
                        const uint32_t to = at + (uint32_t)(((blk * 4 + j) ^ (r & 7)) * 16);
                        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" :: "r"(to), "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3]) : "memory");
                        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" :: "r"(to + (uint32_t)N * 128u), "r"(l[0]), "r"(l[1]), "r"(l[2]), "r"(l[3]) : "memory");
                    }
                    tc_fence_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(s_full + slot);
                    i += turns; slot += turns;
                    if (slot >= S) { slot -= S; phase ^= 1u; }
                };
                load(q[0], sc[0]);
                load(q[1], sc[1]);
                while (i < n_all && ok) {
                    load(q[2], sc[2]); store(q[0], sc[0]);
                    load(q[0], sc[0]); store(q[1], sc[1]);
                    load(q[1], sc[1]); store(q[2], sc[2]);
                }
            }
        }
    } else if (warp < 8) {
        // ================================================================= tokens: a thread has one
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" :: "n"(TS_REGS_X));
        const int wq = warp & 3;
        if (wq < live_quarters && n_tiles) {
            const uint32_t row = (uint32_t)(wq * 32 + lane);
            int ab = 0, xb = 0, slot = 0, free_slot = 0, n = 0;       // slot of this stage, and of the one two before it, which had its buffer
            unsigned free_phase = 0u, xphase = 0u;
            bool ok = true;
            auto lds = [&](uint32_t at) -> uint4 {
                uint4 v;
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
                return v;
            };
            for (int i = 0; i < n_tiles * (n_st / 2) && ok; i++) {
                ok = wait(s_xfull + xb, xphase);
                const uint32_t from = xbufs + (uint32_t)xb * TS_XBUF;
                const uint4 d4 = lds(from + 2 * TS_TOK * 64 + row * 16u);
                const float d[4] = {__uint_as_float(d4.x), __uint_as_float(d4.y), __uint_as_float(d4.z), __uint_as_float(d4.w)};
#pragma unroll
                for (int h = 0; h < 2; h++) {                         // two stages
                    const uint32_t a = tmem + ((uint32_t)(wq * 32) << 16) + TS_A + (uint32_t)ab * 64u;
#pragma unroll
                    for (int b = 0; b < 2; b++) {
                        const uint32_t at = from + row * 64u + (uint32_t)(((2 * h + b) ^ (row >> 1 & 3u)) * 16u);   // (as TMA permutes rows of 64 bytes)
                        const uint4 xl = lds(at), xh = lds(at + TS_TOK * 64);
                        const uint32_t w[8] = {xl.x, xh.x, xl.y, xh.y, xl.z, xh.z, xl.w, xh.w};
                        const float down = large ? __uint_as_float((uint32_t)(127 - ts_down(d[2 * h + b])) << 23) : 1.f;
                        const uint32_t s2 = (uint32_t)__half_as_ushort(__float2half_rn(d[2 * h + b] * down)) * 0x10001u;
                        uint32_t hi16[16], lo16[16];
#pragma unroll
                        for (int j = 0; j < 8; j++) {                 // four int8: 1024 + 128 + v as halves, bytes 0 and 2, then 1 and 3
                            const uint32_t u = w[j] ^ 0x80808080u;
                            ts_split(ts_add2(__byte_perm(u, 0x64646464u, 0x4240), 0xE480E480u), s2, hi16[2 * j], lo16[2 * j]);        // 0xE480 = -1152
                            ts_split(ts_add2(__byte_perm(u, 0x64646464u, 0x4341), 0xE480E480u), s2, hi16[2 * j + 1], lo16[2 * j + 1]);
                        }
                        if (b == 0 && n++ >= 2) {
                            ok = wait(s_empty + free_slot, free_phase) && ok;
                            if (++free_slot == S) { free_slot = 0; free_phase ^= 1u; }
                            tc_fence_after();
                        }
                        tc_st16(a + 16u * b, hi16);
                        tc_st16(a + 32u + 16u * b, lo16);
                    }
                    if (h == 1) {
                        __syncwarp();
                        if (lane == 0) mbar_arrive(s_xempty + xb);
                    }
                    tc_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(s_full + slot);
                    if (++slot == S) slot = 0;
                    ab ^= 1;
                }
                xb ^= 1;
                if (xb == 0) xphase ^= 1u;
            }
        }
    } else {
        // ================================================================= drains
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" :: "n"(TS_REGS_C));
        const int wq = warp & 3, g = (warp >> 2) - 3;                 // quarter of the tokens, half of the columns
        const bool live = wq < live_quarters;
        float acc[TS_NC];
#pragma unroll
        for (int j = 0; j < TS_NC; j++) acc[j] = 0.f;
        int db = 0;
        const int n_drains = large ? p.nb : n_st;                     // of a tile
        unsigned dphase = 0u;
        bool ok = true, odd = false;                                  // (a sum that is not finite)
        const uint32_t mine_at = tmem + ((uint32_t)(wq * 32) << 16) + (uint32_t)(g * nc);
        const float * xd = p.x.d + (size_t)(tok0 + min(wq * 32 + lane, Tt - 1)) * p.nb;
        auto tile_sums = [&](auto pieces) {                           // up to 32, 64 or 80 columns (what lies beyond nc is some other warp's, and dropped)
            constexpr int C = decltype(pieces)::value;
#pragma unroll 1
            for (int st = 0; st < n_drains; st++) {
                const float up = large ? __uint_as_float((uint32_t)(127 + ts_down(xd[st])) << 23) : 1.f;
                ok = wait(s_dfull + db, dphase) && ok;
                tc_fence_after();
                const uint32_t src = mine_at + (uint32_t)db * TS_N;
#pragma unroll
                for (int c = 0; c < C; c += 8) {
                    float v[8];
                    tc_ld8(v, src + c);
                    if (c + 8 == C) {                                 // the buffer goes back
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(s_dempty + db);
                    }
#pragma unroll
                    for (int j = 0; j < 8; j++) acc[c + j] = fmaf(v[j], up, acc[c + j]);
                }
                db ^= 1;
                if (db == 0) dphase ^= 1u;
            }
        };
#pragma unroll 1
        for (int tile = 0; tile < n_tiles && live; tile++) {
            if (nc <= 32)      tile_sums(std::integral_constant<int, 32>());
            else if (nc <= 64) tile_sums(std::integral_constant<int, 64>());
            else               tile_sums(std::integral_constant<int, TS_NC>());
            // ---- the tile is complete: a thread holds one token's rows; 16 items at a time become lanes
            const int n_tile = min(items, hi - lo - tile * items), half = items / 2;
            float * mine = epi + (warp - 12) * (TS_EPI / 4);
#pragma unroll
            for (int j = 0; j < TS_NC; j++) odd |= j < nc && !(fabsf(acc[j]) < __int_as_float(0x7F800000));        // (behind nc: what an earlier kernel left)
#pragma unroll 1
            for (int c = 0; c < half; c += 16) {                      // (one copy of the body: only the selection is unrolled)
                const int k0 = g * half + c;                          // item of the tile
                if (k0 < n_tile && ok) {
#pragma unroll
                    for (int s = 0; s < (GATED ? TS_NC / 2 : TS_NC); s += 16) {
                        if (s != c) continue;
#pragma unroll
                        for (int j = 0; j < 16; j++) {
                            const int k = (s + j) % (TS_NC / 2);
                            mine[j * 34 + lane] = GATED ? fmaxf(acc[2 * k + 1], 0.f) * acc[2 * k] : acc[s + j];
                        }
                    }
                    __syncwarp();
                    const int k = k0 + (lane & 15);
                    if ((lane & 15) + c < half && k < n_tile) {
                        const int item = lo + tile * items + k;
                        const int r = SPARSE ? rows[tile * items + k] : item;
                        const int64_t gid = SPARSE && p.bucket ? p.bucket[r] : r;
                        const float bias = p.bias ? p.bias[gid] : 0.f;
#pragma unroll 1
                        for (int u0 = 0; u0 < 16; u0 += 8) {
                            float l[8];                               // (predictor logits: all on their way before the first is looked at)
#pragma unroll
                            for (int u = 0; u < 8; u++) {
                                const int tok = tok0 + wq * 32 + (u0 + u) * 2 + (lane >> 4);
                                l[u] = SPARSE && tok < p.T ? p.idx[(size_t)tok * p.idx_stride + gid] : 0.f;
                            }
#pragma unroll
                            for (int u = 0; u < 8; u++) {
                                const int tw = (u0 + u) * 2 + (lane >> 4), tok = tok0 + wq * 32 + tw;
                                const bool off = SPARSE && l[u] < p.threshold;        // (a NaN logit counts as active)
                                float o = off ? 0.f : mine[(lane & 15) * 34 + tw];
                                if (p.bias) o += bias;
                                if (p.relu) o = fmaxf(o, 0.f);
                                if (tok < p.T) {
                                    if (p.dst)   p.dst[(size_t)tok * p.dst_stride + gid] = o;
                                    if (p.dst16) p.dst16[(size_t)tok * p.dst_stride + gid] = __float2half_rn(o);
                                }
                            }
                        }
                    }
                    __syncwarp();
                }
            }
#pragma unroll
            for (int j = 0; j < TS_NC; j++) acc[j] = 0.f;
        }
        // ---- rows beyond the halves' range, by the warp that wrote their results: a lane has a token
        if (live && ok && __any_sync(0xffffffffu, odd)) {
            const int tok = tok0 + wq * 32 + lane;
            const size_t xb = (size_t)min(tok, p.T - 1) * p.nb;
#pragma unroll 1
            for (int item = lo; item < hi; item++) {
                if ((item - lo) % items / (items / 2) != g) continue;
                const int r = SPARSE ? rows[item - lo] : item;
                const uint8_t * const row = p.W + (size_t)r * p.row_bytes, * const row2 = GATED ? p.W2 + (size_t)r * p.row_bytes : nullptr;
                if (!ts_row_beyond(row, p.nb, lane) && !(GATED && ts_row_beyond(row2, p.nb, lane))) continue;
                const int64_t gid = SPARSE && p.bucket ? p.bucket[r] : r;
                if (tok >= p.T || (SPARSE && p.idx[(size_t)tok * p.idx_stride + gid] < p.threshold)) continue;
                float o = ts_row_sum(row, p.x.lo + xb, p.x.hi + xb, p.x.d + xb, p.nb);
                if (GATED) o *= fmaxf(ts_row_sum(row2, p.x.lo + xb, p.x.hi + xb, p.x.d + xb, p.nb), 0.f);
                if (p.bias) o += p.bias[gid];
                if (p.relu) o = fmaxf(o, 0.f);
                if (p.dst)   p.dst[(size_t)tok * p.dst_stride + gid] = o;
                if (p.dst16) p.dst16[(size_t)tok * p.dst_stride + gid] = __float2half_rn(o);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tc_dealloc(tmem, 512);
}

// ---------------------------------------------------------------------------------------------- launch
template <bool SPARSE, bool GATED>
static int ts_go(TsP & p, bool pdl, cudaStream_t st) {
    const int G = sm_count();
    p.n_tt = (p.T + TS_TOK - 1) / TS_TOK;
    p.groups = (int)imin64(G / p.n_tt, (p.nrows + 7) / 8);
    const int list = SPARSE ? ((p.nrows + p.groups - 1) / p.groups + 1) * 4 : 0;   // bytes
    p.ring = (int)(TS_SMEM_MAX - 1024 - TS_CONS * TS_EPI - 2 * TS_XBUF - list) / 1024 * 1024;
    if (p.ring < 2 * TS_N * 256) return PI_ERR_UNSUPPORTED;
    static bool attr_done[16] = {false};
    int dev = 0;
    PI_CUDA(cudaGetDevice(&dev));
    auto kern = k_mm_q4<SPARSE, GATED>;
    if (dev >= 0 && dev < 16 && !attr_done[dev]) {
        PI_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TS_SMEM_MAX));
        attr_done[dev] = true;
    }
    PI_CUDA(launch_k(kern, dim3(p.groups * p.n_tt), dim3(TS_THREADS), (size_t)TS_SMEM_MAX, st, pdl, p));
    return PI_OK;
}

// Sums of fewer than 2816 columns are more precise in one chain, or no less (see above).  A CTA's time per 64 columns hardly depends on its rows and not at
// all on its tokens up to 128 (hand-overs; the kernel with mma.sync takes steps of 64, 80, 96, 128, 192 and 256 tokens).  us, pi_mm_wide.cu | here:
//   gathers (whose results it writes token by token, too)   97 tokens 4096 x 4096 60 | 52, 8192 x 8192 120 | 93; 256 tokens 88 | 67, 193 | 124
//   dense, 193 .. 256 tokens   4096 x 4096 61.6 | 54.2, 10240 x 8192 193 | 129; where the rows of a CTA pair are just more than one tile here and those of
//                              a CTA just less than one there (two tiles take twice the time of one, however high) 13824 x 4096 101 | 108,
//                              13824 x 8192 192 | 195: stays there; the next tile there, 14300 x 4096, 151 | 118
//   dense, 129 .. 192          8192 x 8192 114 | 114, 5120 x 5120 75 | 69: stays there
//   dense, 97 .. 128           4096 x 4096 41.8 | 45.5, 8192 x 8192 93 | 90, 10240 x 8192 114 | 103
//   fewer                      10240 x 8192, 77 tokens 83 | 102
bool mm_q4_takes(const GemvArgs & a) {
    if (a.ncols < 2816) return false;
    const int T = a.T > 256 ? 256 : a.T;
    if (a.masks) return T > 96;
    if (T > 192) return a.nrows <= sm_count() / 2 * TS_N || a.nrows > sm_count() * 96;
    return T > 96 && T <= 128 && a.nrows >= 10000;
}

// Called by launch_mm, which has checked the arguments.  Tokens go in launches of at most 256.
int launch_mm_q4(const GemvArgs & a, cudaStream_t st) {
    for (int t0 = 0; t0 < a.T; t0 += 256) {
        TsP p;
        p.W = (const uint8_t *)a.W; p.W2 = (const uint8_t *)a.W2; p.row_bytes = (int64_t)pi_row_bytes(a.wtype, a.ncols);
        p.nrows = (int)a.nrows; p.nb = (int)(a.ncols / 32);
        p.T = a.T - t0 < 256 ? a.T - t0 : 256;
        p.x.lo = a.x.lo + (size_t)t0 * p.nb; p.x.hi = a.x.hi + (size_t)t0 * p.nb; p.x.d = a.x.d + (size_t)t0 * p.nb;
        p.masks = a.masks; p.bucket = a.bucket; p.list = a.list_out; p.count = a.count_out; p.rows_total = t0 == 0 ? a.rows_total : nullptr;
        p.idx = a.idx ? a.idx + (size_t)t0 * a.idx_stride : nullptr; p.idx_stride = a.idx_stride; p.threshold = a.threshold;
        p.bias = a.bias; p.relu = a.relu;
        p.dst = a.dst ? a.dst + (size_t)t0 * a.dst_stride : nullptr;
        p.dst16 = a.dst16 ? a.dst16 + (size_t)t0 * a.dst_stride : nullptr; p.dst_stride = a.dst_stride;
        p.status = a.status;
        int rc;
        if ((rc = tensor_map(&p.m_lo, CU_TENSOR_MAP_DATA_TYPE_UINT8, p.x.lo, (int64_t)p.nb * 16, p.T, (int64_t)p.nb * 16, 64, TS_TOK, CU_TENSOR_MAP_SWIZZLE_64B)) != PI_OK) return rc;
        if ((rc = tensor_map(&p.m_hi, CU_TENSOR_MAP_DATA_TYPE_UINT8, p.x.hi, (int64_t)p.nb * 16, p.T, (int64_t)p.nb * 16, 64, TS_TOK, CU_TENSOR_MAP_SWIZZLE_64B)) != PI_OK) return rc;
        if ((rc = tensor_map(&p.m_d, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, p.x.d, p.nb, p.T, (int64_t)p.nb * 4, 4, TS_TOK, CU_TENSOR_MAP_SWIZZLE_NONE)) != PI_OK) return rc;
        rc = !p.masks ? ts_go<false, false>(p, a.pdl, st) : p.W2 ? ts_go<true, true>(p, a.pdl, st) : ts_go<true, false>(p, a.pdl, st);
        if (rc != PI_OK) return rc;
    }
    return PI_OK;
}

}  // namespace pi
