// Mat-mat over FP16 rows for many tokens on tcgen05: the operators, row selection and epilogue of pi_mm.cu.
//
// Bound: the bytes that an SM brings in, its rows once and all activations (77 tokens of 12288 x 4096: 0.7 MB and 0.6 MB an SM).
//
// Work split: TOKENS are the 128 lanes of the products (M; two tiles of them beyond 128), rows their columns (N, steps of 16), so that every
// CTA takes its equal contiguous range of rows, as in pi_mm.cu: with rows as lanes 96 of 148 SMs would share 12288 rows, and a range of
// few rows would cost as much as 128.  Sums stay in tensor memory until a tile of up to 256 rows has seen all columns.
//
// Warps: 0 brings activations and dense rows as TMA tiles, 1 issues the products, 4..15 write the results: a thread holds ONE token's rows
// after tcgen05.ld, 16 columns at a time become lanes through shared memory.  Gathered rows these warps copy first, through registers (in
// one launch of 8600 of 11008 gated rows of 8 KB: 47 us; rows by cp.async, 50 clocks per warp and copy, 70 in the kernel before this one; by
// tile::gather4, 90 clocks per four rows of 128 bytes, 94).
//
// Short rows are the launch's fixed part: what a CTA finds out before its first request (ranges come from the host, no 64-bit division), the first
// trip to memory, and the results' way out.  us, mma.sync | here, 64 tokens: 1024 x 64 4.4 | 4.7, 512 x 128 4.7 | 4.7, 1024 x 256 5.4 | 5.3.
//
// us, mma.sync | here, 77, 128 and 256 tokens: 12288 x 4096 38.7 | 26.0, 51.5 | 30.2, 74.4 | 37.6; 1024 x 4096 30.2 | 11.5, 38.1 | 11.7, 42.9 | 12.7;
// the FFN of 72 % of 11008 x 4096, down projection included, 119 | 71, 175 | 78, 290 | 118.
#include "pi_tc.cuh"

#include <atomic>
#include <type_traits>

namespace pi {

static constexpr int MT_THREADS = 512, MT_OUT = 384;    // threads 128 .. 511 copy and write
static constexpr int MT_EPI = 16 * 34 * 4;               // a warp's transposition of 16 rows x 32 tokens
static constexpr int MT_SMAX = 8;                        // stages at most
static constexpr int MT_SMEM_MAX = 226 * 1024;
static constexpr int MT_RANKS = 4;                       // CTAs that share the columns of a range of rows (SPLIT)
static constexpr int MT_PASS = MT_OUT / 8;              // rows of a pass of the copying threads

struct alignas(64) MtP {
    CUtensorMap m_w, m_x;
    const uint8_t * W; const uint8_t * W2; int64_t row_bytes; int nrows, ncols;
    int groups, share, more;                                     // groups of CTAs along the rows; dense: rows (masks_out: bytes of the masks) of a group, groups that have one more
    int T, nt, n_tt, x_rows, per_tile, ring;             // token tiles of a CTA (1, 2), CTAs that share rows, rows of an activation box, of a dense box, bytes of the ring
    const uint32_t * masks; const int32_t * bucket; int32_t * list; int32_t * count; unsigned long long * rows_total;
    const float * idx; int64_t idx_stride; float threshold;
    const float * bias; int relu;
    float * dst; __half * dst16; int64_t dst_stride;
    __half * coef; int64_t coef_stride; bool coef_tail;           // zeros behind the last position (k_axpy_tc reads stages of 64)
    uint32_t * masks_out; float masks_threshold; int masks_or;
    unsigned int * status;
};

template <bool SPARSE, bool GATED, bool SPLIT>
__global__ void __launch_bounds__(MT_THREADS, 1) k_mm_tc(const __grid_constant__ MtP p) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ int s_warp[MT_THREADS / 32];
    __shared__ unsigned s_any[8];
    __shared__ uint64_t s_full[MT_SMAX], s_empty[MT_SMAX], s_dfull[2], s_dempty[2], s_fin;
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_dead;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);    // (uniform for the compiler)
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
    float * const epi = reinterpret_cast<float *>(smem_raw + (ring - smem_u32(smem_raw)) + p.ring);
    int * const rows = reinterpret_cast<int *>(epi + MT_OUT / 32 * (MT_EPI / 4));      // rows of this CTA (sparse only)
    constexpr int ks = SPLIT ? MT_RANKS : 1;
    const int rank = SPLIT ? (int)(blockIdx.x % ks) : 0, block = blockIdx.x / ks;       // ranges of columns, this CTA's
    const int cta = p.n_tt == 1 ? block : (int)((unsigned)block / (unsigned)p.n_tt), tok_first = (block - cta * p.n_tt) * p.x_rows;
    const int tok_end = p.n_tt > 1 ? min(p.T, tok_first + p.x_rows) : p.T;
    if (tid == 32) { tma_map(&p.m_x); if (!SPARSE) tma_map(&p.m_w); }
    if (tid < 8) s_any[tid] = 0u;
    if (tid < MT_SMAX) { mbar_init(s_full + tid, SPARSE ? 1 + MT_OUT / 32 : 1); mbar_init(s_empty + tid, 1); }
    if (tid < 2) { mbar_init(s_dfull + tid, 1); mbar_init(s_dempty + tid, MT_OUT / 32); }
    if (tid == 0) { mbar_init(&s_fin, 1); s_dead = 0; }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (warp == 0) tc_alloc(&s_tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem, 0);
    if (SPLIT) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // (waited for before the first store into a neighbour's memory)
    pdl_launch();
    auto wait = [&](uint64_t * bar, unsigned parity) -> bool {        // warp-uniform; false: the wait ran out, here or elsewhere
        bool ok = false;
        for (int spins = 0; spins < (1 << 20) && !ok && !s_dead; spins++) ok = mbar_try_wait(bar, parity);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok && lane == 0) { s_dead = 1; if (p.status) atomicOr(p.status, 16u); }
        return ok;
    };

    int lo, hi;
    if (SPARSE) {
        pdl_wait();
        const int total = tc_active_rows<MT_THREADS>(p.masks, p.nrows, cta, p.groups, s_warp, rows, lo, hi);
        if (blockIdx.x == 0 && tid == 0) {
            if (p.count) *p.count = total;
            if (p.rows_total && total) atomicAdd(p.rows_total, (unsigned long long)total);      // statistics
        }
        if (p.list && tok_first == 0) for (int k = tid; k < hi - lo; k += MT_THREADS) p.list[lo + k] = rows[k];
        if (p.coef_tail && cta == p.groups - 1 && tok_first == 0) {
            const int64_t end = (total + 63) / 64 * 64 < p.coef_stride ? (total + 63) / 64 * 64 : p.coef_stride;
            for (int e = tid; e < p.T * 64; e += MT_THREADS)
                if (total + e % 64 < end) p.coef[(size_t)(e / 64) * p.coef_stride + total + e % 64] = __ushort_as_half((unsigned short)0);
        }
    } else {
        const int al = p.masks_out ? 8 : 1;                           // (a byte of the masks has one writer)
        lo = min(p.nrows, (p.share * cta + min(cta, p.more)) * al);
        hi = min(p.nrows, (p.share * (cta + 1) + min(cta + 1, p.more)) * al);
    }
    // tiles of equal height, N columns each (gated: column pairs, up and gate of one item)
    const int n_cols = (hi - lo) * (GATED ? 2 : 1);
    const int n_tiles = SPARSE ? (n_cols + 255) / 256 : n_cols <= p.per_tile ? n_cols > 0 : (int)((unsigned)(n_cols + p.per_tile - 1) / (unsigned)p.per_tile);
    const int N = SPARSE ? (n_tiles ? ((n_cols + n_tiles - 1) / n_tiles + 15) / 16 * 16 : 16) : (p.per_tile + 15) / 16 * 16;
    const int items = GATED ? N / 2 : SPARSE ? N : p.per_tile;        // of a tile
    const int all_slices = (p.ncols + 63) / 64, slice0 = all_slices * rank / ks;
    const int n_slices = all_slices * (rank + 1) / ks - slice0;
    const int n_bufs = p.nt * N <= 256 ? 2 : 1;
    // A stage is `su` slices of 64 columns, as many as leave three stages: a hand-over costs each of the three parties 200 .. 400 clocks,
    // a slice of few rows less (1024 x 4096, 77 tokens: one slice a stage 23.9 us, four 17.0).
    const uint32_t w_off = p.nt > 1 ? 32768u : (uint32_t)p.x_rows * 128u, slice_bytes = w_off + (uint32_t)N * 128u;
    const int fit = (int)((unsigned)p.ring / slice_bytes), deep = SPARSE ? (N <= 2 * MT_PASS ? 4 : N <= 4 * MT_PASS ? 2 : 1) : 4;   // (gathered: slices that a thread copies at once)
    const int su = min(min(deep, n_slices), fit >= 12 ? 4 : fit >= 6 ? 2 : 1), S = min(MT_SMAX, (int)((unsigned)fit / (unsigned)su)), n_stages = n_slices <= su ? 1 : su == 1 ? n_slices : (int)((unsigned)(n_slices + su - 1) / (unsigned)su);
    const uint32_t stage = slice_bytes * (uint32_t)su;
    if (!SPARSE) pdl_wait();

    if (warp == 0) {
        // ================================================================= TMA tiles
        int slot = 0, slice = 0, row = lo;
        unsigned phase = 1u;                                          // parity of the hand-back to wait for (first round: none)
        int i = 0;
        for (; i < n_tiles * n_stages; i++) {
            if (!wait(s_empty + slot, phase)) break;
            if (lane == 0) {
                mbar_expect_tx(s_full + slot, (unsigned)(su * (p.nt * p.x_rows + (SPARSE ? 0 : p.per_tile)) * 128));
                for (int u = 0; u < su; u++) {
                    const uint32_t base = ring + (uint32_t)slot * stage + (uint32_t)u * slice_bytes;
                    const int col = (SPLIT && slice + u >= n_slices ? all_slices : slice0 + slice + u) * 64;       // (behind the last slice: zeros)
                    for (int t = 0; t < p.nt; t++) tma_tile(base + t * 16384, &p.m_x, col, tok_first + t * 128, s_full + slot);
                    if (!SPARSE) tma_tile(base + w_off, &p.m_w, col, row, s_full + slot);
                }
            }
            __syncwarp();
            slice += su;
            if (slice >= n_slices) { slice = 0; row += items; }
            if (++slot == S) { slot = 0; phase ^= 1u; }
        }
        if (lane == 0) ring_land(s_full, i, S);
        __syncwarp();
    } else if (warp == 1) {
        // ================================================================= products
        const uint32_t idesc = tc_idesc(N, false);
        int slot = 0, buf = 0;
        unsigned phase = 0u, dphase = 1u;                             // (the first tiles' buffers are free)
        bool ok = true;
        for (int tile = 0; tile < n_tiles && ok; tile++) {
            ok = wait(s_dempty + buf, dphase);
            const uint32_t d = tmem + (uint32_t)(buf * 256);
            for (int s = 0; s < n_stages && ok; s++) {
                ok = wait(s_full + slot, phase);
                if (!ok) break;
                tc_fence_after();
                uint32_t at = ring + (uint32_t)slot * stage;
                for (int u = 0; u < su; u++, at += slice_bytes) {
                    const uint64_t a = tc_desc_k(at), w = tc_desc_k(at + w_off);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        tc_mma_f16(d, a + 2 * k, w + 2 * k, idesc, s + u > 0 || k > 0);
                        if (p.nt > 1) tc_mma_f16(d + (uint32_t)N, a + 1024 + 2 * k, w + 2 * k, idesc, s + u > 0 || k > 0);
                    }
                }
                tc_commit(s_empty + slot);
                if (++slot == S) { slot = 0; phase ^= 1u; }
            }
            tc_commit(s_dfull + buf);
            if (++buf == n_bufs) { buf = 0; dphase ^= 1u; }
        }
        tc_commit(&s_fin);                                            // nothing is in flight when tensor memory is given back
        for (int spins = 0; spins < (1 << 20) && !mbar_try_wait(&s_fin, 0u); spins++) {}
        __syncwarp();
    } else if (warp >= 4) {
        const int pt = tid - (MT_THREADS - MT_OUT), quarter = warp & 3, third = (warp >> 2) - 1;
        float * const mine = epi + (warp - 4) * (MT_EPI / 4);
        // (SPLIT) sums of 16 rows x 32 tokens: [rank they come from][group of 16 rows of this CTA][quarter of the tokens][row][token]
        float * const red = epi + MT_OUT / 32 * (MT_EPI / 4);
        const int quarters = (p.x_rows + 31) / 32, red_rank = (N / 16 + ks - 1) / ks * quarters * 512;
        int buf = 0;
        unsigned dphase = 0u;
        bool ok = true;
        // ---- the results of a tile
        auto write = [&](int tile) {
            if (!SPLIT) ok = wait(s_dfull + buf, dphase) && ok;
            tc_fence_after();
            const int n_tile = min(items, hi - lo - tile * items);
            constexpr int PER = GATED ? 8 : 16;                       // items of 16 columns
            for (int t = 0; t < p.nt; t++) {
                const int tok0 = tok_first + t * 128 + quarter * 32;
                if (tok0 >= tok_end) break;
                for (int c = (SPLIT ? third * ks + rank : third) * 16; c < N; c += 48 * ks) {
                    const int k0 = GATED ? c / 2 : c;
                    if (k0 >= n_tile) break;
                    float v[16];
                    if (SPLIT) {                                      // the cluster's sums, in the order of their columns
                        const float * part = red + ((c / 16 / ks) * quarters + quarter) * 512 + lane;
#pragma unroll
                        for (int j = 0; j < 16; j++) v[j] = part[j * 32];
#pragma unroll
                        for (int k = 1; k < ks; k++) {
                            part += red_rank;
#pragma unroll
                            for (int j = 0; j < 16; j++) v[j] += part[j * 32];
                        }
                    } else tc_ld16(v, tmem + (uint32_t)(quarter * 32 << 16) + (uint32_t)(buf * 256 + t * N + c));
                    if (GATED) {
#pragma unroll
                        for (int j = 0; j < 8; j++) mine[j * 34 + lane] = fmaxf(v[2 * j + 1], 0.f) * v[2 * j];
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; j++) mine[j * 34 + lane] = v[j];
                    }
                    __syncwarp();
                    const int kl = lane % PER, k = k0 + kl;
                    bool any = false;
                    if (k < n_tile) {
                        const int item = lo + tile * items + k;
                        const int r = SPARSE ? rows[tile * items + k] : item;
                        const int64_t gid = SPARSE && p.bucket ? p.bucket[r] : r;
                        const float bias = p.bias ? p.bias[gid] : 0.f;
                        if (SPARSE) {
                            float l[PER];                             // (predictor logits: all on their way before the first is looked at)
#pragma unroll
                            for (int u = 0; u < PER; u++) {
                                const int tok = tok0 + u * (32 / PER) + lane / PER;
                                l[u] = tok < tok_end ? p.idx[(size_t)tok * p.idx_stride + gid] : 0.f;
                            }
#pragma unroll
                            for (int u = 0; u < PER; u++) {
                                const int tw = u * (32 / PER) + lane / PER, tok = tok0 + tw;
                                const bool off = l[u] < p.threshold;          // (a NaN logit counts as active)
                                float o = off ? 0.f : mine[kl * 34 + tw];
                                if (p.bias && !(off && p.coef)) o += bias;    // (a coefficient of an inactive token is 0 whatever the bias)
                                if (p.relu) o = fmaxf(o, 0.f);
                                if (tok < tok_end) {
                                    if (p.dst)   p.dst[(size_t)tok * p.dst_stride + gid] = o;
                                    if (p.dst16) p.dst16[(size_t)tok * p.dst_stride + gid] = __float2half_rn(o);
                                    if (p.coef)  p.coef[(size_t)tok * p.coef_stride + item] = __float2half_rn(o);
                                }
                            }
                        } else {
                            // Eight values are there before the first is stored, because a load of shared memory does not pass a store through a
                            // pointer (16 rows of 64 tokens, clocks: one by one 2600, here 900; the gathers, with more to keep, 1.2 times slower so)
#pragma unroll 1
                            for (int u0 = 0; u0 < 32; u0 += 16) {
                                const int tw0 = u0 + (lane >> 4), first = tok0 + tw0, n_tok = tok_end - first;
                                float o[8];
#pragma unroll
                                for (int u = 0; u < 8; u++) {
                                    o[u] = mine[kl * 34 + tw0 + 2 * u];
                                    if (p.bias) o[u] += bias;
                                    if (p.relu) o[u] = fmaxf(o[u], 0.f);
                                    any |= 2 * u < n_tok && !(o[u] < p.masks_threshold);
                                }
                                auto put = [&](auto * to, auto as) {
                                    to += (size_t)first * p.dst_stride + gid;
#pragma unroll
                                    for (int u = 0; u < 8; u++, to += 2 * p.dst_stride) if (2 * u < n_tok) *to = as(o[u]);
                                };
                                if (p.dst)   put(p.dst, [](float v) { return v; });
                                if (p.dst16) put(p.dst16, [](float v) { return __float2half_rn(v); });
                            }
                        }
                        if (!SPARSE && p.masks_out && any) atomicOr(&s_any[k / 32], 1u << (k % 32));
                    }
                    __syncwarp();
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(s_dempty + buf);
            if (++buf == n_bufs) { buf = 0; dphase ^= 1u; }
            if (!SPARSE && p.masks_out) {                             // the union over the tokens of !(result < threshold), one bit per row
                asm volatile("bar.sync 1, 384;" ::: "memory");
                if (pt < 32 && pt * 8 < n_tile) {                     // the range starts at a multiple of 8 rows
                    unsigned char * o = reinterpret_cast<unsigned char *>(p.masks_out) + (lo + tile * items) / 8 + pt;
                    const unsigned char bits = (unsigned char)(s_any[pt / 4] >> (pt % 4 * 8));
                    *o = p.masks_or ? (unsigned char)(*o | bits) : bits;
                }
                __syncwarp();
                if (pt < 8) s_any[pt] = 0u;
                asm volatile("bar.sync 1, 384;" ::: "memory");
            }
        };
        if (SPLIT) {
            // ---- a tile's sums go to the CTA of the cluster that writes these rows
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
            if (n_tiles) {
                ok = wait(s_dfull, 0u);
                tc_fence_after();
                for (int c = third; c < N / 16 && quarter < quarters; c += 3) {
                    float v[16];
                    tc_ld16(v, tmem + (uint32_t)(quarter * 32 << 16) + (uint32_t)(c * 16));
                    uint32_t to;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(smem_u32(red + rank * red_rank + ((c / ks) * quarters + quarter) * 512 + lane)), "r"(c % ks));
#pragma unroll
                    for (int j = 0; j < 16; j++) asm volatile("st.shared::cluster.f32 [%0], %1;" :: "r"(to + (uint32_t)j * 128u), "f"(v[j]) : "memory");
                }
            }
            __syncwarp();
            asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
            if (n_tiles && ok) write(0);
        } else if (!SPARSE) {
            for (int tile = 0; tile < n_tiles; tile++) write(tile);
        } else {
            // ---- gathered rows: 8 threads a row, 48 rows a pass, as many passes as the tile has rows for.  A thread requests 6 .. 9 pieces at once, of U
            // slices, while those before are stored: 36 .. 54 KB on their way per SM (with 96 KB slower: 8600 of 11008 rows of 8 KB, gated, 77 tokens
            // 71 against 60 us).  Nothing is requested for a column of no row: with two, four or eight passes, and some row in the place of
            // those beyond the tile, every CTA asked the L2 for the same lines, up to half of its requests (us, before | here, 77, 128 and 256
            // tokens: idx, 72 % of 4096 x 4096 33.9 | 26.9, 41.9 | 32.5, 50.4 | 43.6; the FFN of 72 % of 11008 x 4096 76.9 | 71.0, 85.0 | 78.1, 123.1 | 117.9).
            auto gather = [&](auto slices, auto passes) {
                constexpr int U = decltype(slices)::value, PJ = decltype(passes)::value, SETS = 2;
                const int piece = pt & 7, r0 = pt >> 3;
                const uint32_t to = (uint32_t)(r0 * 128 + (piece ^ (r0 & 7)) * 16);       // (48 is a multiple of 8: the same place in every pass)
                const int n_steps = (n_stages * su + U - 1) / U;
                int slot = 0;
                unsigned phase = 1u;
#pragma unroll 1
                for (int tile = 0; tile < n_tiles && ok; tile++) {
                    const uint8_t * src[PJ];
#pragma unroll
                    for (int j = 0; j < PJ; j++) {
                        const int r = r0 + j * MT_PASS, k = GATED ? r >> 1 : r, item = tile * items + k;
                        src[j] = k < items && lo + item < hi ? (GATED && (r & 1) ? p.W2 : p.W) + (size_t)rows[item] * p.row_bytes + piece * 16 : nullptr;
                    }
                    uint4 v[SETS][U * PJ];
                    auto load = [&](int step, uint4 (&b)[U * PJ]) {
                        if (step >= n_steps) return;
                        const int x = step * U * 64 + piece * 8;      // (a row's end: zeros)
#pragma unroll
                        for (int u = 0; u < U; u++)
#pragma unroll
                            for (int j = 0; j < PJ; j++) b[u * PJ + j] = src[j] && x + u * 64 < p.ncols ? ldg_stream(src[j] + (size_t)(step * U + u) * 128) : make_uint4(0u, 0u, 0u, 0u);
                    };
                    int part = 0;                                     // slice of the stage
                    auto store = [&](int step, const uint4 (&b)[U * PJ]) {
                        if (step >= n_steps) return;
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            if (step * U + u >= n_stages * su) break;
                            if (part == 0) ok = wait(s_empty + slot, phase) && ok;
                            const uint32_t at = ring + (uint32_t)slot * stage + (uint32_t)part * slice_bytes + w_off + to;
#pragma unroll
                            for (int j = 0; j < PJ; j++)
                                if (r0 + j * MT_PASS < N)
                                    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" :: "r"(at + j * MT_PASS * 128), "r"(b[u * PJ + j].x), "r"(b[u * PJ + j].y), "r"(b[u * PJ + j].z), "r"(b[u * PJ + j].w) : "memory");
                            if (++part < su) continue;
                            part = 0;
                            tc_fence_smem();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(s_full + slot);
                            if (++slot == S) { slot = 0; phase ^= 1u; }
                        }
                    };
#pragma unroll
                    for (int k = 0; k < SETS - 1; k++) load(k, v[k]);
#pragma unroll 1
                    for (int i = 0; i < n_steps && ok; i += SETS) {
#pragma unroll
                        for (int k = 0; k < SETS; k++) {
                            load(i + k + SETS - 1, v[(k + SETS - 1) % SETS]);
                            store(i + k, v[k]);
                        }
                    }
                    write(tile);
                }
            };
            if (N <= MT_PASS)          gather(std::integral_constant<int, 8>(), std::integral_constant<int, 1>());
            else if (N <= 2 * MT_PASS) gather(std::integral_constant<int, 4>(), std::integral_constant<int, 2>());
            else if (N <= 3 * MT_PASS) gather(std::integral_constant<int, 3>(), std::integral_constant<int, 3>());
            else if (N <= 4 * MT_PASS) gather(std::integral_constant<int, 2>(), std::integral_constant<int, 4>());
            else                       gather(std::integral_constant<int, 1>(), std::integral_constant<int, 6>());
        }
        tc_fence_before();
    }
    if (SPLIT && warp < 4) {                                          // (the two barriers of the cluster, for the warps that write nothing)
        __syncwarp();
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tc_dealloc(tmem, 512);
}

// ---------------------------------------------------------------------------------------------- launch
static cudaLaunchConfig_t mt_config(int clusters, cudaLaunchAttribute * attr, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(clusters * MT_RANKS); cfg.blockDim = dim3(MT_THREADS); cfg.dynamicSmemBytes = MT_SMEM_MAX; cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = MT_RANKS; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    return cfg;
}

// clusters that this device keeps resident at once (B200: 33)
static int mt_clusters() {
    static std::atomic<int> known[16];
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return 0;
    if ((n = known[dev].load()) > 0) return n;
    auto kern = k_mm_tc<false, false, true>;
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = mt_config(1, attr, nullptr);
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MT_SMEM_MAX) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    known[dev].store(n);
    return n;
}

template <bool SPARSE, bool GATED, bool SPLIT>
static int mt_go(MtP & p, bool pdl, cudaStream_t st) {
    const int G = SPLIT ? mt_clusters() / p.n_tt : (int)imin64(sm_count() / p.n_tt, (p.nrows + 7) / 8);
    const int list = SPARSE ? ((p.nrows + G - 1) / G + 1) * 4 : 0;    // bytes
    p.ring = (MT_SMEM_MAX - 1024 - MT_OUT / 32 * MT_EPI - list) / 1024 * 1024;
    if (p.ring < 2 * (p.nt * 16384 + 256 * 128)) return PI_ERR_UNSUPPORTED;        // two stages of the largest kind (more than MM_MAX_ROWS rows)
    p.groups = G; p.per_tile = 0;
    int rc;
    if (!SPARSE) {                                                    // equal tiles; whole bytes of the masks
        // (dealt out here: a division of 64 bits takes a CTA 0.2 us)
        const int units = p.masks_out ? (p.nrows + 7) / 8 : p.nrows;
        p.share = units / G; p.more = units % G;
        const int share = (p.nrows + G - 1) / G + (p.masks_out ? 8 : 0), tiles = (share + 255) / 256;
        p.per_tile = p.masks_out ? (share / tiles + 8) / 8 * 8 : (share + tiles - 1) / tiles;
        if (p.per_tile > 256) p.per_tile = 256;
        if ((rc = tensor_map(&p.m_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, p.W, p.ncols, p.nrows, p.row_bytes, 64, p.per_tile, CU_TENSOR_MAP_SWIZZLE_128B)) != PI_OK) return rc;
    }
    if (SPLIT) p.ring -= ((p.per_tile + 15) / 16 + MT_RANKS) * ((p.x_rows + 31) / 32) * 2048 / 1024 * 1024;      // what comes from the cluster
    static bool attr_done[16] = {false};
    int dev = 0;
    PI_CUDA(cudaGetDevice(&dev));
    auto kern = k_mm_tc<SPARSE, GATED, SPLIT>;
    if (dev >= 0 && dev < 16 && !attr_done[dev]) {
        PI_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MT_SMEM_MAX));
        attr_done[dev] = true;
    }
    if (!SPLIT) { PI_CUDA(launch_k(kern, dim3(G * p.n_tt), dim3(MT_THREADS), (size_t)MT_SMEM_MAX, st, pdl, p)); return PI_OK; }
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = mt_config(G * p.n_tt, attr, st);
    cfg.numAttrs = pdl ? 2 : 1;
    PI_CUDA(cudaLaunchKernelEx(&cfg, kern, (const MtP &)p));
    return PI_OK;
}

// Called by launch_mm, which has checked the arguments.  Tokens go in launches of at most 256.
int launch_mm_tc(const GemvArgs & a, cudaStream_t st) {
    for (int t0 = 0; t0 < a.T; t0 += 256) {
        MtP p;
        p.W = (const uint8_t *)a.W; p.W2 = (const uint8_t *)a.W2; p.row_bytes = a.ncols * 2;
        p.nrows = (int)a.nrows; p.ncols = (int)a.ncols;
        p.T = a.T - t0 < 256 ? a.T - t0 : 256;
        // Dense rows: all CTAs have all of the tokens, or groups of n neighbours have a part of them each (64 at least) and n times the rows.  What a
        // CTA brings in decides: its tokens, and its r rows one and a half times (us, 256 tokens, n = 1 | 2 | 3 | 4: 4096 x 4096 32.7 | 24.3 | 24.8 | 26.2,
        // 12288 x 4096 41.5 | 37.5 | 45.7 | 55.8; 128 tokens, n = 1 | 2: 8192 x 8192 38.0 | 37.6, 12288 x 4096 29.9 | 35.1).  Two token tiles in one
        // CTA cost their products, too: 44 more.
        // Few rows leave a CTA the activations and a chain of column slices, 0.2 us each whatever they hold: four CTAs of a cluster then take a
        // quarter of the columns each, of four times the rows, up to 160 in a CTA (so that a part of the tokens still is 64 or more), and add up their
        // sums through each other's shared memory.  us, in a graph, alone | in fours, 77, 128, 256 tokens: 1024 x 4096 16.5 | 11.5, 16.6 | 11.7, 17.2 |
        // 12.7; 1024 x 8192 26.8 | 15.0, 27.1 | 15.2, 29.1 | 17.8; 2048 x 2048 11.3 | 10.1, 11.6 | 11.0, 13.3 | 12.3; 4096 x 4096 16.9 | 14.4, 18.4 | 14.8; 5120 x
        // 5120 19.8 | 16.5, 25.5 | 19.4; no gain below 2048 columns (2048 x 1024 8.7 | 9.1).  In pairs 13.0 for the first, 8192 x 8192 36.2 | 35.3, 38.0 | 39.4.
        // Gathered rows go through the CTA's registers, so that doing it twice costs more (idx, 72 % of 2048 x 2048 40 | 35, 4096 x 4096 64 | 50, 11008 x
        // 1024 54 | 57).  Masks are the union over ALL tokens.
        p.n_tt = 1;
        bool split = false;
        if (a.masks) p.n_tt = p.T > 128 && a.nrows * (a.W2 ? 2 : 1) < 6000 ? 2 : 1;
        else if (!a.masks_out) {
            for (int n = p.T > 128 ? p.T / 64 : 1; n >= (p.T + 127) / 128 && a.ncols >= 2048 && !split; n--) {
                const int G = mt_clusters() / n;
                if (G > 0 && (a.nrows + G - 1) / G <= 160) { split = true; p.n_tt = n; }
            }
            auto brought = [&](int n) { return (n == 1 && p.T > 128 ? 300 : ((p.T + n - 1) / n + 7) / 8 * 8) + 3 * a.nrows * n / (2 * sm_count()); };
            for (int n = 2; n <= p.T / 64 && !split; n++) if (brought(n) < brought(p.n_tt)) p.n_tt = n;
        }
        p.x_rows = ((p.T + p.n_tt - 1) / p.n_tt + 7) / 8 * 8;
        if (p.x_rows > 128) p.x_rows = 128;
        p.nt = p.n_tt > 1 ? 1 : (p.T + 127) / 128;
        if (p.n_tt > 1) p.n_tt = (p.T + p.x_rows - 1) / p.x_rows;
        int rc = tensor_map(&p.m_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a.x.h16 + (size_t)t0 * a.ncols, p.ncols, p.T, (int64_t)p.ncols * 2, 64, p.x_rows, CU_TENSOR_MAP_SWIZZLE_128B);
        if (rc != PI_OK) return rc;
        p.masks = a.masks; p.bucket = a.bucket; p.list = a.list_out; p.count = a.count_out; p.rows_total = t0 == 0 ? a.rows_total : nullptr;
        p.idx = a.idx ? a.idx + (size_t)t0 * a.idx_stride : nullptr; p.idx_stride = a.idx_stride; p.threshold = a.threshold;
        p.bias = a.bias; p.relu = a.relu;
        p.dst = a.dst ? a.dst + (size_t)t0 * a.dst_stride : nullptr;
        p.dst16 = a.dst16 ? a.dst16 + (size_t)t0 * a.dst_stride : nullptr; p.dst_stride = a.dst_stride;
        p.coef = a.coef ? a.coef + (size_t)t0 * a.coef_stride : nullptr; p.coef_stride = a.coef_stride; p.coef_tail = a.coef && a.T > AXPY_TC_TOKENS;
        p.masks_out = a.masks_out; p.masks_threshold = a.masks_threshold; p.masks_or = t0 > 0; p.status = a.status;
        rc = split ? mt_go<false, false, true>(p, a.pdl, st) : !p.masks ? mt_go<false, false, false>(p, a.pdl, st) : p.W2 ? mt_go<true, true, false>(p, a.pdl, st) : mt_go<true, false, false>(p, a.pdl, st);
        if (rc != PI_OK) return rc;
    }
    return PI_OK;
}

}  // namespace pi
