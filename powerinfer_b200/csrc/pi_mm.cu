// Small-batch mat-mat (2..32 tokens) over FP16 and planar Q4_0 rows: the dense products and the gather behind
// ggml_mul_mat_idx (with the gate rows riding along), every weight read once for all tokens of the step.
//
// Bound: HBM, as at one token, as long as three other costs stay under the 23 bytes per clock that an SM's share of HBM
// delivers.  (1) The activation slices that a tile needs travel from L2 beside its weights: a tile of 128 rows adds 25 % at
// 32 tokens where a tile of 16 rows adds 200 %.  (2) The products: mma.sync.m16n8k16 (FP16 x FP16 -> FP32, the products of two
// halves are exact) issues at 955 multiply-adds per clock and SM, 8.6 of the 22 clocks that 16 x 16 weights take to arrive
// at 32 tokens; m16n8k32 (s8 x s8 -> s32) at 1990.  (3) Q4_0 scales every block of 32 columns by its own FP32 factor, as the
// CPU path does: three FP32 operations per row, token and block, 12.4 of 12.5 clocks at 32 tokens (at 8 tokens 3.1).
//
// Work split: every CTA (one per SM) takes an equal contiguous range of rows, to the row, whatever their number: no last wave, and
// no two CTAs meet in a tile.  (Equal ranges of K slices with the partial sums added by the last CTA to come cost 10-15 us
// per launch in fences and round trips.)  A range is cut into equal tiles of at most TM rows; the fragment rows that a tile
// leaves unused carry whatever shared memory holds and are never stored, as are the unused token columns.
// The rows of a gather are named by the union of the tokens' activity masks (one bit per neuron): every CTA scans the few
// KB of masks itself and takes the rows of its ranks, so no list has to be built first; it leaves its part of the list behind
// for the axpy.  A dense product can write such masks (the predictor's second matrix does): no mask kernel in between.
//
// Inside a CTA 8 consumer warps split the COLUMNS: a warp takes every eighth slice of 64 bytes of all rows of the tile, and the
// activation of that slice, from a ring of its own that a producer warp of its own fills.  Nothing is shared while a tile lasts, and
// there is no barrier between the first slice and the last, where the 8 partial tiles meet in shared memory and are added in warp
// order.  (16 warps that shared a stage met in a barrier for each: 1900 clocks a stage, whatever it held.  Warps that issued their own
// copies spent half of the time in them: a cp.async waits while the SM's queue of outstanding loads is full, which with HBM as the
// bound is always.)  Consumers get 200 registers, 128 of them accumulators, producers 56.
// Rows arrive by 16-byte cp.async: the rows of the active list lie anywhere, and pieces of a few hundred bytes are too small for the
// bulk-copy engine (about 80 ns per copy).  A row slice of 64 bytes is stored with its four 16-byte pieces permuted by
// (row / 2) % 4, so that the eight rows of an 8x8 fragment lie in different banks without padding.
// Dense weights do not depend on the kernel before: the producers request their first stages before griddepcontrol.wait, and every thread
// waits there before its first bounded wait.
// Every wait is bounded: when one runs out the warp sets bit 4 of *status (where given) and the CTA returns without a result, its copies landed.
//
// Q4_0 arithmetic: a nibble q is placed in the high half of a byte and its top bit flipped, which is the int8 value
// 16 * (q - 8): one logic operation for four weights, no correction term.  The mma's C operand is the constant 0x4B400000, so
// the accumulator comes out as the bits of the float 12582912 + 16 * dot and one subtraction replaces the conversion (exact:
// |16 * dot| <= 520192 < 2^22); the factor 1/16 goes into the weight's scale.
#include "pi_common.cuh"

namespace pi {

static constexpr int MM_RINGS = 8, MM_WARPS = 2 * MM_RINGS, MM_THREADS = MM_WARPS * 32;      // consumer warps 0 .. 7, producer warps 8 .. 15
static constexpr int MM_REGS_C = 200, MM_REGS_P = 56;   // 256 x (200 + 56) = the 512 x 128 of the launch
static constexpr int MM_SMAX = 8;                       // stages of a ring at most
static constexpr int MM_SMEM_MAX = 225 * 1024;          // (leaves room for the static variables)
static constexpr int MM_SLACK = 4096;                   // behind the last ring: fragments past a tile read up to 48 rows (3072 bytes, 384 of scales) on

struct MmP {
    const uint8_t * W; const uint8_t * W2; int64_t row_bytes; int nrows, ncols, nb;
    Act x; int T;
    const uint32_t * masks; const int32_t * bucket; int32_t * list; int32_t * count; unsigned long long * rows_total;
    const float * idx; int64_t idx_stride; float threshold;
    const float * bias; int relu;
    float * dst; __half * dst16; int64_t dst_stride; float * const * dst_host;
    __half * coef; int64_t coef_stride;
    uint32_t * masks_out; float masks_threshold;
    unsigned int * status;
    int n_slices, ring;                                               // slices of 64 bytes of a row; bytes of a warp's ring
};

__device__ __forceinline__ void mm_cp16(uint32_t dst, const void * src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void mm_zero16(uint32_t dst) { asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" :: "r"(dst), "r"(0u) : "memory"); }
__device__ __forceinline__ void mm_cp4(uint32_t dst, const void * src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void mm_cp8(uint32_t dst, const void * src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" :: "r"(dst), "l"(src) : "memory");
}
// one arrival on `bar` when all copies this thread has issued so far have landed
__device__ __forceinline__ void mm_arrive_copies(uint64_t * bar) { asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" :: "r"(smem_u32(bar)) : "memory"); }
__device__ __forceinline__ void mm_ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mm_hmma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mm_imma(uint32_t (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, uint32_t c) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c));
}
__device__ __forceinline__ unsigned long long mm_pack(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ unsigned long long mm_packu(uint32_t a, uint32_t b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ unsigned long long mm_mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// acc += (v * dd - magic * dd) * d4, two tokens at a time.  The first factor is (v - magic) * dd rounded once: dd holds 11 bits
// (an FP16 number), so magic * dd = 1.5 * 2^23 * dd is exact.
__device__ __forceinline__ void mm_scale_add(unsigned long long & acc, unsigned long long v, unsigned long long dd, unsigned long long md, unsigned long long d4) {
    asm("{\n .reg .b64 t;\n fma.rn.f32x2 t, %1, %2, %3;\n fma.rn.f32x2 %0, t, %4, %0;\n}" : "+l"(acc) : "l"(v), "l"(dd), "l"(md), "l"(d4));
}

template <int WT, int NT>
struct MmShape {
    static constexpr bool Q4 = WT == PI_TYPE_Q4_0;
    static constexpr int TP = NT * 8;                                 // token rows of a stage
    static constexpr int MT = Q4 && NT == 4 ? 7 : 8;                  // fragments of 16 rows of a tile at most (two stages have to fit)
    // Fragments that are multiplied without a branch between them: a branch around every fragment left each one's chain of latencies
    // (fragment, nibbles, product, scale: 150 clocks) in the open.  Few tokens leave the pipes idle anyway: fragments of 16 rows that
    // the tile does not have are then cheaper multiplied (their rows are whatever lies behind the tile) than skipped.
    static constexpr int MG = NT <= 2 ? 4 : 2, MA = (MT + MG - 1) / MG * MG;
    static constexpr int KS = Q4 ? 128 : 32;                          // columns of a slice
    static constexpr int ROW = Q4 ? 72 : 64, TOK = Q4 ? 144 : 64;     // bytes of a stage per row and per token
    static_assert(2 * (MT * 16 * ROW + TP * TOK) * MM_RINGS <= MM_SMEM_MAX - 8192 - MM_SLACK, "two stages");
};

template <int WT, int NT, bool SPARSE, bool GATED>
__global__ void __launch_bounds__(MM_THREADS, 1) k_mm(const MmP p) {
    using Z = MmShape<WT, NT>;
    constexpr bool Q4 = Z::Q4;
    constexpr int TP = Z::TP, MT = Z::MT, MG = Z::MG, MA = Z::MA;
    constexpr int IT = GATED ? MT * 8 : MT * 16;                      // items (rows / neurons) of a tile at most
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_warp[MM_WARPS];
    __shared__ unsigned s_any[4];
    __shared__ uint64_t s_full[MM_RINGS][MM_SMAX], s_empty[MM_RINGS][MM_SMAX], s_tile;
    __shared__ volatile int s_dead;
    int * rows = reinterpret_cast<int *>(smem + (size_t)MM_RINGS * p.ring);      // rows of this CTA (sparse only)
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);    // (a shuffle: uniform for the compiler too; a branch it takes for divergent costs every mma behind it)
    const int G = gridDim.x, cta = blockIdx.x;
    const int me = warp & (MM_RINGS - 1);                             // my ring
    const uint32_t ring_a = smem_u32(smem) + (uint32_t)(me * p.ring);
    uint64_t * full = s_full[me], * empty = s_empty[me];
    pdl_launch();
    if (tid < MM_RINGS * MM_SMAX) { mbar_init(&s_full[0][0] + tid, 64); mbar_init(&s_empty[0][0] + tid, 1); }
    if (tid == 0) { mbar_init(&s_tile, MM_RINGS); s_dead = 0; }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncthreads();
    auto wait = [&](uint64_t * bar, unsigned parity) -> bool {        // warp-uniform; false: the wait ran out, here or elsewhere
        bool ok = false;
        for (int spins = 0; spins < (1 << 20) && !ok && !s_dead; spins++) ok = mbar_try_wait(bar, parity);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok && lane == 0) { s_dead = 1; if (p.status) atomicOr(p.status, 16u); }
        return ok;
    };

    // this CTA's items, items per tile, fragment rows of a tile, bytes of a stage, stages of a ring
    int lo = 0, hi = 0, per_tile = 1, n_tiles = 0, rt = 16, stage = 1, S = 2;
    auto set_range = [&](int n) {
        const int al = !SPARSE && p.masks_out ? 8 : 1;                // (a byte of the masks has one writer)
        const int gr = (n + al - 1) / al;
        lo = min(n, (int)((long long)gr * cta / G) * al);
        hi = min(n, (int)((long long)gr * (cta + 1) / G) * al);
        n_tiles = (hi - lo + IT - 1) / IT;
        if (n_tiles > 0) per_tile = ((hi - lo + n_tiles - 1) / n_tiles + al - 1) / al * al;
        rt = ((GATED ? 2 * per_tile : per_tile) + 15) / 16 * 16;
        stage = rt * Z::ROW + TP * Z::TOK;
        S = min(MM_SMAX, p.ring / stage);
    };
    const int n_mine = me < p.n_slices ? (p.n_slices - me + MM_RINGS - 1) / MM_RINGS : 0;       // slices of a tile that are mine
    // A stage: row slices, activation slices (Q4_0: then the rows' scales and the activation's, [block][token])
    int first = 0, n_rows = 0;                                        // current tile: first item, rows in all (gated: up 0, gate 0, up 1, ..)
    const int r8 = lane >> 2, c4 = lane & 3;
    const uint32_t w_dst = (uint32_t)(r8 * 64 + ((c4 ^ (r8 >> 1)) & 3) * 16);
    auto row_ptr = [&](int r) -> const uint8_t * {
        const int k = GATED ? r >> 1 : r;
        return (GATED && (r & 1) ? p.W2 : p.W) + (size_t)(SPARSE ? rows[first + k] : lo + first + k) * p.row_bytes;
    };
    // Addresses are kept and moved along: a producer is one warp, and a chain of address arithmetic per copy costs it more than the copy.
    const bool ragged = !Q4 && p.ncols % 32 != 0;                     // the last slice of a row is not whole
    const uint8_t * w_src = nullptr; const uint8_t * s_src = nullptr; // dense: my piece of row r8 (Q4_0: my scales of row `lane`) of the next slice
    const size_t w_step = (size_t)p.row_bytes * 8, s_step = (size_t)p.row_bytes * 32;
    auto issue_w = [&](int j, int slot) {                             // my slice number j (asked for in order within a tile)
        const int s = me + j * MM_RINGS;
        const uint32_t base = ring_a + (uint32_t)(slot * stage), to = base + w_dst;
        const int off = s * 64 + c4 * 16;
        if (!SPARSE && j == 0) { w_src = row_ptr(r8) + off; if (Q4) s_src = row_ptr(lane) + (size_t)p.nb * 16 + s * 8; }
        if (ragged && off >= p.ncols * 2) {                           // past the end of a row: zeros
            for (int r = r8; r < n_rows; r += 8) mm_zero16(to + (r - r8) * 64);
            __threadfence_block();
        } else if (!SPARSE) {
            const uint8_t * src = w_src;
#pragma unroll 4
            for (int r = r8; r < n_rows; r += 8, src += w_step) mm_cp16(to + (r - r8) * 64, src);
        } else {
#pragma unroll 4
            for (int r = r8; r < n_rows; r += 8) mm_cp16(to + (r - r8) * 64, row_ptr(r) + off);
        }
        w_src += 64 * MM_RINGS;
        if (Q4) {
            const uint32_t sb = base + rt * 64 + TP * 128;
            const int so = p.nb * 16 + s * 8;
            const uint8_t * src = s_src;
            for (int r = lane; r < n_rows; r += 32, src += s_step) mm_cp8(sb + r * 8, SPARSE ? row_ptr(r) + so : src);
            s_src += 8 * MM_RINGS;
        }
    };
    // The activation of a slice: 16-byte pieces, 8 (Q4_0: 4) tokens per instruction.  Columns of tokens past the last one keep whatever shared
    // memory holds, like the rows past a tile: no product mixes columns.  (Filled with the last token's bytes they cost what its lines
    // cost at the L2, which every CTA asks for at once: 10240 x 8192 Q4_0, 2 tokens 30.7 us where it is 18.4, 8 tokens 18.9.)
    constexpr int XN = Q4 ? 2 * NT : NT, XT = Q4 ? 4 : 8;             // instructions, tokens of one
    const int xr = Q4 ? lane >> 3 : r8, xc = Q4 ? lane & 7 : c4;
    const uint32_t x_dst = Q4 ? (uint32_t)(xr * 128 + ((xc ^ xr) & 7) * 16) : (uint32_t)(xr * 64 + ((xc ^ (xr >> 1)) & 3) * 16);
    int x_at[XN], d_at[Q4 ? NT : 1];                                  // byte offsets of my tokens
    const char * x_src = Q4 ? reinterpret_cast<const char *>((xc & 1 ? p.x.hi : p.x.lo) + (xc >> 1)) : reinterpret_cast<const char *>(p.x.h16 + xc * 8);
    const char * d_src = reinterpret_cast<const char *>(p.x.d) + (lane & 3) * 4;
    auto start_x = [&]() {
#pragma unroll
        for (int i = 0; i < XN; i++) x_at[i] = (xr + i * XT) * (Q4 ? p.nb * 16 : p.ncols * 2);
#pragma unroll
        for (int i = 0; i < (Q4 ? NT : 0); i++) d_at[i] = ((lane >> 2) + i * 8) * p.nb * 4;
    };
    auto issue_x = [&](int j, int slot) {
        const int s = me + j * MM_RINGS;
        const uint32_t base = ring_a + (uint32_t)(slot * stage + rt * 64), to = base + x_dst;
        if (ragged && s * 32 + xc * 8 >= p.ncols) {
#pragma unroll
            for (int i = 0; i < XN; i++) mm_zero16(to + i * 512);
            __threadfence_block();
        } else {
            const char * src = x_src + s * 64;
#pragma unroll
            for (int i = 0; i < XN; i++) if (xr + i * XT < p.T) mm_cp16(Q4 && (i & 1) ? (to + i * 512) ^ 64u : to + i * 512, src + x_at[i]);      // (token + 4: piece ^ 4)
        }
        if (Q4) {
            const uint32_t dt = base + TP * 128 + rt * 8 + ((lane & 3) * TP + (lane >> 2)) * 4;
#pragma unroll
            for (int i = 0; i < (Q4 ? NT : 0); i++) if ((lane >> 2) + i * 8 < p.T) mm_cp4(dt + i * 32, d_src + s * 16 + d_at[i]);
        }
    };
    auto start_tile = [&](int tile) {
        first = tile * per_tile;
        n_rows = min(per_tile, hi - lo - first) * (GATED ? 2 : 1);
    };

    if (!SPARSE) {
        set_range(p.nrows);
    } else {
        pdl_wait();
        // ---- ranks of the active rows: thread t counts the words [c0, c1), a block scan gives the rank of its first row
        constexpr int KEEP = 4;
        const int n_chunks = (p.nrows + 31) / 32, per = (n_chunks + MM_THREADS - 1) / MM_THREADS;
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
        for (int w = 0; w < MM_WARPS; w++) { if (w < warp) before += s_warp[w]; total += s_warp[w]; }
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
        if (p.list) for (int k = tid; k < hi - lo; k += MM_THREADS) p.list[lo + k] = rows[k];
    }

    if (warp >= MM_RINGS) {
        // ================================================================= producers
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" :: "n"(MM_REGS_P));
        start_x();
        int slot = 0, ahead = 0;                                      // ahead: stages of tile 0 requested before the loop
        unsigned phase = 1u;                                          // parity of the hand-back to wait for (first round: none)
        if (!SPARSE) {
            start_tile(0);
            const int ns = n_tiles > 0 ? min(S, n_mine) : 0;
            for (int j = 0; j < ns; j++) { issue_w(j, j); mm_arrive_copies(full + j); }
            pdl_wait();
            for (int j = 0; j < ns; j++) { issue_x(j, j); mm_arrive_copies(full + j); }
            ahead = ns;
            slot = ns == S ? 0 : ns;
            if (ns == S) phase = 0u;
        }
        for (int tile = 0; tile < n_tiles; tile++) {
            start_tile(tile);
            if (tile > 0 && !wait(&s_tile, (unsigned)(tile - 1) & 1u)) break;      // the sums of the tile before lie over the rings
            bool ok = true;
            for (int j = tile == 0 ? ahead : 0; j < n_mine; j++) {
                ok = wait(empty + slot, phase);
                if (!ok) break;
                issue_w(j, slot);
                mm_arrive_copies(full + slot);
                issue_x(j, slot);
                mm_arrive_copies(full + slot);
                if (++slot == S) { slot = 0; phase ^= 1u; }
            }
            if (!ok) break;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        return;
    }
    // ===================================================================== consumers
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" :: "n"(MM_REGS_C));
    // The waits below are bounded in tries: they count this kernel's own copies only, not what is left of the kernel before (an exchange may
    // wait for a late rank for a second), and do not take issue slots from it.
    if (!SPARSE) pdl_wait();
    const int g = lane >> 2, q = lane & 3;
    // ldmatrix addresses inside a stage (fragment layouts of mma.m16n8k16 / m16n8k32): two 16-byte pieces of 16 rows, four of 8 tokens
    // (Q4_0: one block of 32 rows, one block of two groups of 8 tokens)
    const int a_row = Q4 ? lane : lane & 15;
    const uint32_t b_up = NT > 1 ? (lane >> 4) * 8 * 128 : 0;
    const int b_row = Q4 ? (lane & 7) + (NT > 1 ? (lane >> 4) * 8 : 0) : (lane & 7);
    const uint32_t MAGIC = 0x4B400000u;
    const unsigned long long neg_magic = mm_pack(-12582912.0f, -12582912.0f), sixteenth = mm_pack(0.0625f, 0.0625f);
    uint32_t a_off[Q4 ? 4 : 2], b_off[Q4 ? 4 : 1];
#pragma unroll
    for (int k = 0; k < (Q4 ? 4 : 2); k++) a_off[k] = (uint32_t)(a_row * 64 + (((Q4 ? k : k * 2 + (lane >> 4)) ^ ((lane & 7) >> 1)) & 3) * 16);
#pragma unroll
    for (int k = 0; k < (Q4 ? 4 : 1); k++)
        b_off[k] = Q4 ? (uint32_t)(b_row * 128 + (((k * 2 + ((lane >> 3) & 1)) ^ (lane & 7)) & 7) * 16) : (uint32_t)(b_row * 64 + (((lane >> 3) ^ ((lane & 7) >> 1)) & 3) * 16);

    int slot = 0;
    unsigned phase = 0u;
    for (int tile = 0; tile < n_tiles; tile++) {
        start_tile(tile);
        // (the accumulators of the two types have different shapes)
        float acc[Q4 ? 1 : MA][Q4 ? 1 : NT][4];
        unsigned long long acq[Q4 ? MA : 1][Q4 ? NT : 1][2];
#pragma unroll
        for (int m = 0; m < MA; m++)
#pragma unroll
            for (int n = 0; n < NT; n++)
#pragma unroll
                for (int j = 0; j < 4; j++) { if (Q4) acq[Q4 ? m : 0][Q4 ? n : 0][j >> 1] = 0ull; else acc[Q4 ? 0 : m][Q4 ? 0 : n][j] = 0.f; }
        for (int i = 0; i < n_mine; i++) {
            if (!wait(full + slot, phase)) break;
            const uint32_t base = ring_a + (uint32_t)(slot * stage), xb = base + rt * 64;
            if (!Q4) {
                uint32_t b[NT][4];
#pragma unroll
                for (int n = 0; n < NT; n++) mm_ldsm4(b[n], xb + b_off[0] + n * 8 * 64);
#pragma unroll
                for (int m0 = 0; m0 < MA; m0 += MG) {
                    if (m0 * 16 >= rt) break;
                    uint32_t a[MG][2][4];
#pragma unroll
                    for (int m = 0; m < MG; m++)
#pragma unroll
                        for (int k = 0; k < 2; k++) mm_ldsm4(a[m][k], base + a_off[k] + (m0 + m) * 16 * 64);
#pragma unroll
                    for (int k = 0; k < 2; k++)
#pragma unroll
                        for (int m = 0; m < MG; m++)
#pragma unroll
                            for (int n = 0; n < NT; n++) mm_hmma(acc[Q4 ? 0 : m0 + m][Q4 ? 0 : n], a[m][k], b[n][2 * k], b[n][2 * k + 1]);
                }
            } else {
                const uint32_t sb = xb + TP * 128 + g * 8, db = xb + TP * 128 + rt * 8 + 2 * q * 4;
#pragma unroll
                for (int m0 = 0; m0 < (Q4 ? MA : 0); m0 += MG) {
                    if (m0 * 16 >= rt) break;
                    uint2 sc[MG][2];                                  // scales of the slice's four blocks, rows g and g + 8
#pragma unroll
                    for (int m = 0; m < MG; m++)
#pragma unroll
                        for (int h = 0; h < 2; h++)
                            asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(sc[m][h].x), "=r"(sc[m][h].y) : "r"(sb + (m0 + m) * 128 + h * 64));
#pragma unroll
                    for (int k = 0; k < 4; k++) {                     // block by block
                        uint32_t w[MG][2], b[NT + 1][2];
                        unsigned long long dd[NT], md[NT];
#pragma unroll
                        for (int m = 0; m < MG; m += 2) {
                            uint32_t v[4];
                            mm_ldsm4(v, base + a_off[k] + (m0 + m) * 16 * 64);
                            w[m][0] = v[0]; w[m][1] = v[1]; w[m + 1][0] = v[2]; w[m + 1][1] = v[3];
                        }
#pragma unroll
                        for (int n = 0; n < NT; n += 2) {
                            uint32_t v[4];
                            mm_ldsm4(v, xb + b_off[k] + n * 8 * 128 - (n + 1 < NT ? 0u : b_up));      // (an odd last group is read twice)
                            b[n][0] = v[0]; b[n][1] = v[1]; b[n + 1][0] = v[2]; b[n + 1][1] = v[3];
                        }
#pragma unroll
                        for (int n = 0; n < NT; n++) {
                            asm volatile("ld.shared.b64 %0, [%1];" : "=l"(dd[n]) : "r"(db + (k * TP + n * 8) * 4));
                            dd[n] = mm_mul2(dd[n], sixteenth);
                            md[n] = mm_mul2(dd[n], neg_magic);
                        }
#pragma unroll
                        for (int m = 0; m < MG; m++) {
                            const float2 f0 = h2f(k < 2 ? sc[m][0].x : sc[m][0].y), f1 = h2f(k < 2 ? sc[m][1].x : sc[m][1].y);
                            const float e0 = k & 1 ? f0.y : f0.x, e1 = k & 1 ? f1.y : f1.x;
                            const unsigned long long d0 = mm_pack(e0, e0), d1 = mm_pack(e1, e1);
                            const uint32_t a0 = ((w[m][0] << 4) & 0xF0F0F0F0u) ^ 0x80808080u, a1 = ((w[m][1] << 4) & 0xF0F0F0F0u) ^ 0x80808080u;
                            const uint32_t a2 = (w[m][0] & 0xF0F0F0F0u) ^ 0x80808080u, a3 = (w[m][1] & 0xF0F0F0F0u) ^ 0x80808080u;
#pragma unroll
                            for (int n = 0; n < NT; n++) {
                                uint32_t c[4];
                                mm_imma(c, a0, a1, a2, a3, b[n][0], b[n][1], MAGIC);
                                mm_scale_add(acq[Q4 ? m0 + m : 0][Q4 ? n : 0][0], mm_packu(c[0], c[1]), dd[n], md[n], d0);
                                mm_scale_add(acq[Q4 ? m0 + m : 0][Q4 ? n : 0][1], mm_packu(c[2], c[3]), dd[n], md[n], d1);
                            }
                        }
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + slot);                 // handed back
            if (++slot == S) { slot = 0; phase ^= 1u; }
        }
        // ---- the warps' partial tiles: [token][row], each over its own ring (all copies have landed: the last stage was the last
        // one requested); a pitch of 4 (20) mod 32 words keeps the fragment stores free of bank conflicts
        const int pitch = rt + 4;
        float * mine = reinterpret_cast<float *>(smem + (size_t)me * p.ring);
#pragma unroll
        for (int m = 0; m < MT; m++) {
            if (m * 16 >= rt) break;
#pragma unroll
            for (int n = 0; n < NT; n++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    float v;
                    if (Q4) {
                        const unsigned long long w = acq[Q4 ? m : 0][Q4 ? n : 0][j >> 1];
                        v = __uint_as_float(j & 1 ? (unsigned)(w >> 32) : (unsigned)w);
                    } else {
                        v = acc[Q4 ? 0 : m][Q4 ? 0 : n][j];
                    }
                    mine[(n * 8 + 2 * q + (j & 1)) * pitch + m * 16 + g + (j >> 1) * 8] = v;
                }
        }
        if (tid < 4) s_any[tid] = 0u;
        {                                                             // all partial tiles are there; the warps agree whether a wait ran out
            int dead = s_dead;
            asm volatile("{\n .reg .pred p, q;\n setp.ne.s32 p, %0, 0;\n bar.red.or.pred q, 1, 256, p;\n selp.s32 %0, 1, 0, q;\n}" : "+r"(dead) :: "memory");
            if (dead) return;
        }
        const float * sums = reinterpret_cast<const float *>(smem);
        const int n_tile = GATED ? n_rows / 2 : n_rows;
        float * const host = !SPARSE && p.dst_host ? *p.dst_host : nullptr;
        for (int k0 = 0; k0 < n_tile; k0 += 32) {                     // a lane per item; tokens warp, warp + 8, ... at once
            const int k = min(k0 + lane, n_tile - 1);
            const bool mine_k = k0 + lane < n_tile;
            const int item = lo + first + k;
            const int r = SPARSE ? rows[first + k] : item;
            const int64_t gid = SPARSE && p.bucket ? p.bucket[r] : r;
            const float bias = p.bias ? p.bias[gid] : 0.f;
            float l[NT], o[NT];
#pragma unroll
            for (int u = 0; u < NT; u++) { const int t = warp + u * 8; l[u] = SPARSE && t < p.T ? p.idx[(size_t)t * p.idx_stride + gid] : 0.f; }
#pragma unroll
            for (int u = 0; u < NT; u++) {
                const int t = warp + u * 8;                           // (sums of tokens past the last are read, and dropped)
                if (GATED) {
                    float up = 0.f, gt = 0.f;
#pragma unroll
                    for (int w = 0; w < MM_RINGS; w++) {
                        const float2 f = *reinterpret_cast<const float2 *>(sums + (size_t)w * (p.ring / 4) + t * pitch + 2 * k);
                        up += f.x; gt += f.y;
                    }
                    o[u] = fmaxf(gt, 0.f) * up;
                } else {
                    o[u] = 0.f;
#pragma unroll
                    for (int w = 0; w < MM_RINGS; w++) o[u] += sums[(size_t)w * (p.ring / 4) + t * pitch + k];
                }
            }
            bool any = false;
#pragma unroll
            for (int u = 0; u < NT; u++) {
                const int t = warp + u * 8;
                if (!mine_k || t >= p.T) continue;
                const bool off = SPARSE && l[u] < p.threshold;        // (a NaN logit counts as active)
                float v = off ? 0.f : o[u];
                if (p.bias) v += bias;
                if (p.relu) v = fmaxf(v, 0.f);
                if (p.dst)   p.dst[(size_t)t * p.dst_stride + gid] = v;
                if (host)    host[(size_t)t * p.dst_stride + gid] = v;
                if (p.dst16) p.dst16[(size_t)t * p.dst_stride + gid] = __float2half_rn(v);
                if (p.coef)  p.coef[(size_t)t * p.coef_stride + item] = __float2half_rn(off ? 0.f : v);
                any |= !(v < p.masks_threshold);
            }
            if (!SPARSE && p.masks_out) {                             // the union over the tokens of !(result < threshold), one bit per row
                const unsigned m = __ballot_sync(0xffffffffu, any);
                if (lane == 0 && m) atomicOr(&s_any[k0 / 32], m);
            }
        }
        if (!SPARSE && p.masks_out) {
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (tid < 16 && tid * 8 < n_tile) {                       // the range starts at a multiple of 8 rows
                unsigned char * o = reinterpret_cast<unsigned char *>(p.masks_out) + (lo + first) / 8 + tid;
                const unsigned char bits = (unsigned char)(s_any[tid / 4] >> (tid % 4 * 8));
                *o = bits;
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&s_tile);                          // the sums are read: when all warps are here the rings may fill again
    }
}

// ---------------------------------------------------------------------------------------------- launch
template <int WT, int NT, bool SPARSE, bool GATED>
static int mm_go(MmP p, bool pdl, cudaStream_t st) {
    using Z = MmShape<WT, NT>;
    p.n_slices = (p.ncols + Z::KS - 1) / Z::KS;
    // (8 rows are as little as is worth a CTA: its share of the activation costs more than its weights)
    const int G = (int)imin64(sm_count(), (p.nrows + 7) / 8);
    const int list = SPARSE ? ((p.nrows + G - 1) / G + 1) * 4 : 0;    // bytes
    if (list > 8192 - 128) return PI_ERR_UNSUPPORTED;                 // (more than MM_MAX_ROWS rows)
    p.ring = (MM_SMEM_MAX - list - MM_SLACK) / MM_RINGS / 128 * 128;
    static bool attr_done[16] = {false};
    int dev = 0;
    PI_CUDA(cudaGetDevice(&dev));
    auto kern = k_mm<WT, NT, SPARSE, GATED>;
    if (dev >= 0 && dev < 16 && !attr_done[dev]) {
        PI_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MM_SMEM_MAX));
        attr_done[dev] = true;
    }
    PI_CUDA(launch_k(kern, dim3(G), dim3(MM_THREADS), (size_t)p.ring * MM_RINGS + list + MM_SLACK, st, pdl, p));
    return PI_OK;
}

template <int WT, int NT>
static int mm_sel(const MmP & p, bool pdl, cudaStream_t st) {
    if (!p.masks) return mm_go<WT, NT, false, false>(p, pdl, st);
    if (p.W2)     return mm_go<WT, NT, true, true>(p, pdl, st);
    return mm_go<WT, NT, true, false>(p, pdl, st);
}

template <int WT>
static int mm_tokens(const MmP & p, bool pdl, cudaStream_t st) {
    if (p.T <= 8)  return mm_sel<WT, 1>(p, pdl, st);
    if (p.T <= 16) return mm_sel<WT, 2>(p, pdl, st);
    if (p.T <= 24) return mm_sel<WT, 3>(p, pdl, st);
    return mm_sel<WT, 4>(p, pdl, st);
}

// PI_ERR_UNSUPPORTED: shape not eligible, the caller uses another kernel.
int launch_mm(const GemvArgs & a, cudaStream_t st) {
    const bool q4 = a.wtype == PI_TYPE_Q4_0;
    if (q4 ? !a.x.lo || a.ncols % 256 != 0 : !a.x.h16 || a.ncols % 8 != 0) return PI_ERR_UNSUPPORTED;
    if (a.nrows > (a.masks ? MM_MAX_ROWS : (1 << 26)) || (a.W2 && !a.masks) || (a.list && !a.masks)) return PI_ERR_UNSUPPORTED;
    if (a.T > 32 && q4 && (a.masks_out || a.coef)) return PI_ERR_UNSUPPORTED;           // (predictors and coefficients as products are FP16 rows')
    if (a.T > 32) return !q4 ? launch_mm_tc(a, st) : mm_q4_takes(a) ? launch_mm_q4(a, st) : launch_mm_wide(a, st);
    MmP p;
    p.W = (const uint8_t *)a.W; p.W2 = (const uint8_t *)a.W2; p.row_bytes = (int64_t)pi_row_bytes(a.wtype, a.ncols);
    p.nrows = (int)a.nrows; p.ncols = (int)a.ncols; p.nb = (int)(a.ncols / 32); p.x = a.x; p.T = a.T;
    p.masks = a.masks; p.bucket = a.bucket; p.list = a.list_out; p.count = a.count_out; p.rows_total = a.rows_total;
    p.idx = a.idx; p.idx_stride = a.idx_stride; p.threshold = a.threshold; p.bias = a.bias; p.relu = a.relu;
    p.dst = a.dst; p.dst16 = a.dst16; p.dst_stride = a.dst_stride; p.dst_host = a.dst_host; p.coef = a.coef; p.coef_stride = a.coef_stride;
    p.masks_out = a.masks_out; p.masks_threshold = a.masks_threshold; p.status = a.status; p.n_slices = 0; p.ring = 0;
    return q4 ? mm_tokens<PI_TYPE_Q4_0>(p, a.pdl, st) : mm_tokens<PI_TYPE_F16>(p, a.pdl, st);
}

}  // namespace pi
