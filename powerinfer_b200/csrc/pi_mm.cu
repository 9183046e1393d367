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
// Inside a CTA 16 warps share a stage: TM / 32 groups of 32 rows, the others split the stage's columns; their sums meet in
// shared memory at the end of a tile, in warp order.  Rows arrive by 16-byte cp.async from all threads: the rows of the active
// list lie anywhere, and pieces of a few hundred bytes are too small for the bulk-copy engine (about 80 ns per copy).
// Dense weights do not depend on the kernel before: their first stages are requested before griddepcontrol.wait.
//
// Q4_0 arithmetic: a nibble q is placed in the high half of a byte and its top bit flipped, which is the int8 value
// 16 * (q - 8): one logic operation for four weights, no correction term.  The mma's C operand is the constant 0x4B400000, so
// the accumulator comes out as the bits of the float 12582912 + 16 * dot and one subtraction replaces the conversion (exact:
// |16 * dot| <= 520192 < 2^22); the factor 1/16 goes into the weight's scale.
#include "pi_common.cuh"

namespace pi {

static constexpr int MM_THREADS = 512, MM_WARPS = 16;
static constexpr int MM_RED_PITCH = 36;                 // floats between tokens of a warp's sums: conflict-free fragment stores
static constexpr size_t MM_SMEM_MAX = 226 * 1024;       // (leaves room for the static variables)

struct MmP {
    const uint8_t * W; const uint8_t * W2; int64_t row_bytes; int nrows, ncols, nb;
    Act x; int T;
    const uint32_t * masks; const int32_t * bucket; int32_t * list; int32_t * count; unsigned long long * rows_total;
    const float * idx; int64_t idx_stride; float threshold;
    const float * bias; int relu;
    float * dst; __half * dst16; int64_t dst_stride;
    __half * coef; int64_t coef_stride;
    uint32_t * masks_out; float masks_threshold; int masks_or;
    int n_slices, max_rows;
};

__device__ __forceinline__ void mm_cp16(uint32_t dst, const void * src, unsigned bytes) {       // the first `bytes` bytes, the rest zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mm_cp4(uint32_t dst, const void * src, unsigned bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" :: "r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mm_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void mm_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }
__device__ __forceinline__ void mm_ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mm_ldsm2(uint32_t & r0, uint32_t & r1, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(addr));
}
__device__ __forceinline__ void mm_hmma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mm_imma(uint32_t (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, uint32_t c) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
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
// acc += (v - magic) * dd * d4, two tokens at a time (each lane of the pair rounds like the scalar operation)
__device__ __forceinline__ void mm_scale_add(unsigned long long & acc, unsigned long long v, unsigned long long neg_magic, unsigned long long dd, unsigned long long d4) {
    asm("{\n .reg .b64 t;\n add.rn.f32x2 t, %1, %2;\n mul.rn.f32x2 t, t, %3;\n fma.rn.f32x2 %0, t, %4, %0;\n}" : "+l"(acc) : "l"(v), "l"(neg_magic), "l"(dd), "l"(d4));
}

template <int WT, int NT, int TM>
struct MmShape {
    static constexpr bool Q4 = WT == PI_TYPE_Q4_0;
    static constexpr int TP = NT * 8;                                 // token rows of a stage
    static constexpr int WM = TM / 32, WK = MM_WARPS / WM;            // warps along the rows, along the columns
    static constexpr int KPW = Q4 ? 2 : ((TM < 128 && NT == 4) || (TM == 32 && NT == 2) ? 1 : 2);   // 16-column steps (32-column blocks) of a warp per stage
    static constexpr int NBS = KPW * WK;                              // steps / blocks of a stage
    static constexpr int KS = NBS * (Q4 ? 32 : 16);
    static constexpr int W_RAW = Q4 ? NBS * 18 : KS * 2;
    static constexpr int W_PITCH = (W_RAW / 16) % 2 ? W_RAW : W_RAW + 16;              // odd multiples of 16 bytes: conflict-free ldmatrix
    static constexpr int X_PITCH = Q4 ? NBS * 32 + 16 : KS * 2 + 16;
    static constexpr int X_OFF = TM * W_PITCH, D_OFF = X_OFF + TP * X_PITCH;
    static constexpr int STAGE = (D_OFF + (Q4 ? NBS * TP * 4 : 0) + 127) / 128 * 128;
    static constexpr int RED = 4 * TP * MM_RED_PITCH * 4;             // sums of 4 warps
    static constexpr int FIT = (int)((MM_SMEM_MAX - 8192 - RED) / STAGE);
    static constexpr int S = FIT > 8 ? 8 : FIT;
    static_assert(S >= 3, "ring too small");
};

template <int WT, int NT, int TM, bool SPARSE, bool GATED>
__global__ void __launch_bounds__(MM_THREADS, 1) k_mm(const MmP p) {
    using Z = MmShape<WT, NT, TM>;
    constexpr bool Q4 = Z::Q4;
    constexpr int TP = Z::TP, WM = Z::WM, WK = Z::WK, KPW = Z::KPW, NBS = Z::NBS, KS = Z::KS, S = Z::S;
    constexpr int IT = GATED ? TM / 2 : TM;                           // items (rows / neurons) of a tile
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_warp[MM_WARPS];
    float * red = reinterpret_cast<float *>(smem);                    // [4][TP][MM_RED_PITCH]
    unsigned char * ring = smem + Z::RED;
    int * rows = reinterpret_cast<int *>(ring + (size_t)S * Z::STAGE);   // [max_rows] rows of this CTA (sparse only)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wk = warp % WK, wm = warp / WK;                         // (warps w and w + 4 share a scheduler: rows a tile leaves unused idle on all four)
    const int G = gridDim.x, cta = blockIdx.x;
    const uint32_t ring_a = smem_u32(ring);
    pdl_launch();

    int lo = 0, hi = 0, per_tile = 1, n_units = 0;                    // this CTA's items, items per tile
    auto set_range = [&](int n) {
        const int al = !SPARSE && p.masks_out ? 8 : 1;                // (a byte of the masks has one writer)
        const int gr = (n + al - 1) / al;
        lo = min(n, (int)((long long)gr * cta / G) * al);
        hi = min(n, (int)((long long)gr * (cta + 1) / G) * al);
        const int tiles = (hi - lo + IT - 1) / IT;
        if (tiles > 0) per_tile = ((hi - lo + tiles - 1) / tiles + al - 1) / al * al;
        n_units = tiles * p.n_slices;
    };
    // ---- copies.  A thread's pieces of a stage lie in the same rows for a whole tile: it keeps their addresses and moves them along.
    constexpr int CH = Q4 ? NBS : KS / 8;                             // 16-byte pieces of a row slice (Q4_0: of its nibbles)
    constexpr int NW = TM * CH / MM_THREADS;                          // pieces per thread
    constexpr int CS = Q4 ? NBS / 8 : 1;                              // Q4_0: pieces of 8 scales
    constexpr int XP = Q4 ? TP * NBS * 2 : TP * CH;                   // activation pieces of a stage
    constexpr int NX = (XP + MM_THREADS - 1) / MM_THREADS;
    static_assert(MM_THREADS % CH == 0 && (TM * CH) % MM_THREADS == 0 && TM * CS <= MM_THREADS && (XP % MM_THREADS == 0 || NX == 1), "copy map");
    const int c16 = tid % CH;                                         // my piece of a row
    const uint8_t * wp[NW]; const uint8_t * sp = p.W;
    unsigned w_ok = 0u;
    int i_tile = 0, i_slice = 0;                                      // the unit that is requested next
    auto tile_start = [&]() {
        const int first = i_tile * per_tile, n_tile = min(per_tile, hi - lo - first);
        auto row_ptr = [&](int r, bool & ok) -> const uint8_t * {
            const int k = GATED ? r % IT : r;
            ok = k < n_tile;
            const int row = ok ? (SPARSE ? rows[first + k] : lo + first + k) : 0;
            return (GATED && r >= IT ? p.W2 : p.W) + (size_t)row * p.row_bytes;
        };
        w_ok = 0u;
#pragma unroll
        for (int j = 0; j < NW; j++) {
            bool ok;
            wp[j] = row_ptr(tid / CH + j * (MM_THREADS / CH), ok) + c16 * 16;
            if (ok) w_ok |= 1u << j;
        }
        if (Q4 && tid < TM * CS) {
            bool ok;
            sp = row_ptr(tid / CS, ok) + (size_t)p.nb * 16 + (tid % CS) * 16;
            if (ok) w_ok |= 1u << NW;
        }
    };
    auto issue_w = [&](int slot) {
        if (i_slice == 0) tile_start();
        const uint32_t base = ring_a + (uint32_t)slot * Z::STAGE + (tid / CH) * Z::W_PITCH + c16 * 16;
        const int have = (Q4 ? p.nb : p.ncols / 8) - i_slice * CH;    // pieces of a row from this slice on
        const unsigned bytes = c16 < have ? 16u : 0u;                 // past the end of a row: zeros
#pragma unroll
        for (int j = 0; j < NW; j++) {
            if (w_ok >> j & 1u) mm_cp16(base + j * (MM_THREADS / CH) * Z::W_PITCH, bytes ? wp[j] : p.W, bytes);
            wp[j] += CH * 16;
        }
        if (Q4) {
            if (w_ok >> NW & 1u) {
                const bool in = (tid % CS) * 8 < have;
                mm_cp16(ring_a + (uint32_t)slot * Z::STAGE + (tid / CS) * Z::W_PITCH + NBS * 16 + (tid % CS) * 16, in ? sp : p.W, in ? 16u : 0u);
            }
            sp += NBS * 2;
        }
    };
    auto issue_x = [&](int slot) {
        const uint32_t base = ring_a + (uint32_t)slot * Z::STAGE;
#pragma unroll
        for (int j = 0; j < NX; j++) {
            const int e = tid + j * MM_THREADS;
            if (!Q4) {
                const int t = e / CH, c = i_slice * CH + c16;         // (512 is a multiple of CH: the piece is c16 again)
                const bool in = c * 8 < p.ncols;
                if (t < p.T) mm_cp16(base + Z::X_OFF + t * Z::X_PITCH + c16 * 16, p.x.h16 + (in ? (size_t)t * p.ncols + c * 8 : 0), in ? 16u : 0u);
            } else {
                const int h = e % 2, c = (e / 2) % NBS, t = e / (2 * NBS), b = i_slice * NBS + c;
                const bool in = b < p.nb;
                if (t < p.T) mm_cp16(base + Z::X_OFF + t * Z::X_PITCH + c * 32 + h * 16, (h ? p.x.hi : p.x.lo) + (in ? (size_t)t * p.nb + b : 0), in ? 16u : 0u);
            }
        }
        if (Q4) {
#pragma unroll
            for (int j = 0; j < (TP * NBS + MM_THREADS - 1) / MM_THREADS; j++) {
                const int e = tid + j * MM_THREADS, c = e % NBS, t = e / NBS, b = i_slice * NBS + c;
                const bool in = b < p.nb;
                if (t < p.T) mm_cp4(base + Z::D_OFF + (c * TP + t) * 4, p.x.d + (in ? (size_t)t * p.nb + b : 0), in ? 4u : 0u);
            }
        }
    };
    auto advance = [&]() { if (++i_slice == p.n_slices) { i_slice = 0; i_tile++; } };

    if (!SPARSE) {
        set_range(p.nrows);
        for (int s = 0; s < S - 1; s++) { if (s < n_units) { issue_w(s); advance(); } mm_commit(); }
        pdl_wait();
        // The activation of the stages requested so far: plain loads, several in flight (as cp.async it would belong to a
        // later group than all the weights above, and the first stage would be waiting for the last)
        const int ns = min(S - 1, n_units);
        constexpr int UN = 4;
        const int PER = Q4 ? p.T * NBS * 2 : p.T * (KS / 8);
        for (int e0 = tid; e0 < ns * PER; e0 += UN * MM_THREADS) {
            uint4 v[UN];
            uint32_t to[UN];
#pragma unroll
            for (int j = 0; j < UN; j++) {
                const int ea = e0 + j * MM_THREADS, s = ea / PER, e = ea % PER, sl = s % p.n_slices;
                v[j] = make_uint4(0u, 0u, 0u, 0u);
                to[j] = 0u;
                if (ea >= ns * PER) continue;
                if (Q4) {
                    const int h = e % 2, c = (e / 2) % NBS, t = e / (2 * NBS), b = sl * NBS + c;
                    to[j] = ring_a + s * Z::STAGE + Z::X_OFF + t * Z::X_PITCH + c * 32 + h * 16;
                    if (b < p.nb) v[j] = (h ? p.x.hi : p.x.lo)[(size_t)t * p.nb + b];
                } else {
                    const int t = e / (KS / 8), c = e % (KS / 8), col = sl * KS + c * 8;
                    to[j] = ring_a + s * Z::STAGE + Z::X_OFF + t * Z::X_PITCH + c * 16;
                    if (col < p.ncols) v[j] = *reinterpret_cast<const uint4 *>(p.x.h16 + (size_t)t * p.ncols + col);
                }
            }
#pragma unroll
            for (int j = 0; j < UN; j++)
                if (e0 + j * MM_THREADS < ns * PER) asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" :: "r"(to[j]), "r"(v[j].x), "r"(v[j].y), "r"(v[j].z), "r"(v[j].w) : "memory");
        }
        if (Q4) {
            const int PD = p.T * NBS;
            for (int e0 = tid; e0 < ns * PD; e0 += UN * MM_THREADS) {
                float v[UN];
#pragma unroll
                for (int j = 0; j < UN; j++) {
                    const int ea = e0 + j * MM_THREADS, s = ea / PD, e = ea % PD, sl = s % p.n_slices, c = e % NBS, t = e / NBS, b = sl * NBS + c;
                    v[j] = ea < ns * PD && b < p.nb ? p.x.d[(size_t)t * p.nb + b] : 0.f;
                }
#pragma unroll
                for (int j = 0; j < UN; j++) {
                    const int ea = e0 + j * MM_THREADS, s = ea / PD, e = ea % PD, c = e % NBS, t = e / NBS;
                    if (ea < ns * PD) asm volatile("st.shared.f32 [%0], %1;" :: "r"(ring_a + s * Z::STAGE + Z::D_OFF + (c * TP + t) * 4), "f"(v[j]) : "memory");
                }
            }
        }
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
        set_range(total);
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
        for (int s = 0; s < S - 1; s++) { if (s < n_units) { issue_w(s); issue_x(s); advance(); } mm_commit(); }
        if (p.list) for (int k = tid; k < hi - lo; k += MM_THREADS) p.list[lo + k] = rows[k];
    }

    constexpr int NA = Q4 ? 1 : 2;                                    // (the accumulators of the two types have different shapes)
    float acc[NA == 2 ? 2 : 1][NA == 2 ? NT : 1][4];
    unsigned long long acq[Q4 ? 2 : 1][Q4 ? NT : 1][2];
    auto clear = [&]() {
        if (Q4) {
#pragma unroll
            for (int m = 0; m < (Q4 ? 2 : 1); m++)
#pragma unroll
                for (int n = 0; n < (Q4 ? NT : 1); n++) { acq[m][n][0] = 0ull; acq[m][n][1] = 0ull; }
        } else {
#pragma unroll
            for (int m = 0; m < (Q4 ? 1 : 2); m++)
#pragma unroll
                for (int n = 0; n < (Q4 ? 1 : NT); n++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[m][n][j] = 0.f;
        }
    };
    clear();
    const int g = lane >> 2, q = lane & 3;
    // ldmatrix row addresses inside a stage (fragment layouts of mma.m16n8k16 / m16n8k32)
    const uint32_t a_off = Q4 ? (uint32_t)((wm * 32 + lane) * Z::W_PITCH + wk * KPW * 16)
                              : (uint32_t)((wm * 32 + (lane & 7) + ((lane >> 3) & 1) * 8) * Z::W_PITCH + (wk * KPW * 16 + (lane >> 4) * 8) * 2);
    const uint32_t s_off = (uint32_t)((wm * 32 + g) * Z::W_PITCH + NBS * 16 + wk * KPW * 2);
    const uint32_t b_off = Q4 ? (uint32_t)(Z::X_OFF + (lane & 7) * Z::X_PITCH + wk * KPW * 32 + (lane >> 3) * 16)
                              : (uint32_t)(Z::X_OFF + ((lane & 7) + (NT > 1 ? ((lane >> 4) & 1) * 8 : 0)) * Z::X_PITCH + (wk * KPW * 16 + ((lane >> 3) & 1) * 8) * 2);
    const uint32_t d_off = (uint32_t)(Z::D_OFF + (wk * KPW * TP + 2 * q) * 4);
    const uint32_t MAGIC = 0x4B400000u;
    const unsigned long long neg_magic = mm_pack(-12582912.0f, -12582912.0f);

    int tile = 0, slice = 0;
    for (int i = 0; i < n_units; i++) {
        mm_wait<S - 2>();
        __syncthreads();                                              // stage i has landed for everybody; stage i - 1 is consumed
        if (i + S - 1 < n_units) { const int slot = (i + S - 1) % S; issue_w(slot); issue_x(slot); advance(); }
        mm_commit();
        const uint32_t base = ring_a + (uint32_t)(i % S) * Z::STAGE;
        const bool busy = (GATED ? wm * 32 % IT : wm * 32) < min(per_tile, hi - lo - tile * per_tile);      // my rows exist
        if (!busy) {
        } else if (!Q4) {
#pragma unroll
            for (int k = 0; k < KPW; k++) {
                uint32_t a[2][4];
                mm_ldsm4(a[0], base + a_off + k * 32);
                mm_ldsm4(a[1], base + a_off + 16 * Z::W_PITCH + k * 32);
                if (NT == 1) {
                    uint32_t b0, b1;
                    mm_ldsm2(b0, b1, base + b_off + k * 32);
                    mm_hmma(acc[0][0], a[0], b0, b1);
                    mm_hmma(acc[NA - 1][0], a[1], b0, b1);
                } else {
#pragma unroll
                    for (int n = 0; n < NT; n += 2) {
                        uint32_t b[4];
                        mm_ldsm4(b, base + b_off + n * 8 * Z::X_PITCH + k * 32);
                        mm_hmma(acc[0][Q4 ? 0 : n], a[0], b[0], b[1]);
                        mm_hmma(acc[NA - 1][Q4 ? 0 : n], a[1], b[0], b[1]);
                        mm_hmma(acc[0][Q4 ? 0 : n + 1], a[0], b[2], b[3]);
                        mm_hmma(acc[NA - 1][Q4 ? 0 : n + 1], a[1], b[2], b[3]);
                    }
                }
            }
        } else {
            // scales of the warp's two blocks, rows g, g + 8, g + 16, g + 24 of its 32
            unsigned long long d4[2][4];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                uint32_t w;
                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w) : "r"(base + s_off + r * 8 * Z::W_PITCH));
                const float2 f = h2f(w);
                d4[0][r] = mm_pack(f.x * 0.0625f, f.x * 0.0625f);
                d4[1][r] = mm_pack(f.y * 0.0625f, f.y * 0.0625f);
            }
            uint32_t al[2][4], ah[2][4];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                uint32_t w[4];
                mm_ldsm4(w, base + a_off + k * 16);
#pragma unroll
                for (int r = 0; r < 4; r++) { al[k][r] = ((w[r] << 4) & 0xF0F0F0F0u) ^ 0x80808080u; ah[k][r] = (w[r] & 0xF0F0F0F0u) ^ 0x80808080u; }
            }
#pragma unroll
            for (int n = 0; n < NT; n++) {
                uint32_t b[4];
                mm_ldsm4(b, base + b_off + n * 8 * Z::X_PITCH);
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    unsigned long long dd;
                    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(dd) : "r"(base + d_off + (k * TP + n * 8) * 4));
#pragma unroll
                    for (int m = 0; m < 2; m++) {
                        uint32_t c[4];
                        mm_imma(c, al[k][2 * m], al[k][2 * m + 1], ah[k][2 * m], ah[k][2 * m + 1], b[2 * k], b[2 * k + 1], MAGIC);
                        mm_scale_add(acq[Q4 ? m : 0][Q4 ? n : 0][0], mm_packu(c[0], c[1]), neg_magic, dd, d4[k][2 * m]);
                        mm_scale_add(acq[Q4 ? m : 0][Q4 ? n : 0][1], mm_packu(c[2], c[3]), neg_magic, dd, d4[k][2 * m + 1]);
                    }
                }
            }
        }
        if (slice == p.n_slices - 1) {
            // ---- the warps' sums meet in shared memory: warps of one round write different slots, rounds in order
            constexpr int SLOTS = WK / 4;
            float * mine = red + (size_t)(wm * SLOTS + wk % SLOTS) * (TP * MM_RED_PITCH);
#pragma unroll 1
            for (int r = 0; r < 4; r++) {
                if (wk / SLOTS == r) {
#pragma unroll
                    for (int m = 0; m < 2; m++)
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
                                float * o = mine + (n * 8 + 2 * q + (j & 1)) * MM_RED_PITCH + m * 16 + g + (j >> 1) * 8;
                                *o = r == 0 ? v : *o + v;
                            }
                }
                __syncthreads();
            }
            auto sum_of = [&](int r, int t) {                         // row r of the tile, token t: slots in order
                const float * o = red + (size_t)(r >> 5) * SLOTS * (TP * MM_RED_PITCH) + t * MM_RED_PITCH + (r & 31);
                float v = o[0];
#pragma unroll
                for (int s = 1; s < SLOTS; s++) v += o[(size_t)s * (TP * MM_RED_PITCH)];
                return v;
            };
            const int first = tile * per_tile, n_tile = min(per_tile, hi - lo - first);
            for (int e = tid; e < IT * p.T; e += MM_THREADS) {
                const int k = e % IT, t = e / IT;                     // item k of the tile
                if (k >= n_tile) continue;
                const int item = lo + first + k;
                const int r = SPARSE ? rows[first + k] : item;
                const int64_t gid = SPARSE && p.bucket ? p.bucket[r] : r;
                const float v = sum_of(k, t);
                float o = GATED ? fmaxf(sum_of(IT + k, t), 0.f) * v : v;
                if (SPARSE && p.idx[(size_t)t * p.idx_stride + gid] < p.threshold) {      // (a NaN logit counts as active)
                    if (p.coef) { p.coef[(size_t)t * p.coef_stride + item] = __ushort_as_half((unsigned short)0); continue; }
                    o = 0.f;
                }
                if (p.bias) o += p.bias[gid];
                if (p.relu) o = fmaxf(o, 0.f);
                if (p.dst)   p.dst[(size_t)t * p.dst_stride + gid] = o;
                if (p.dst16) p.dst16[(size_t)t * p.dst_stride + gid] = __float2half_rn(o);
                if (p.coef)  p.coef[(size_t)t * p.coef_stride + item] = __float2half_rn(o);
            }
            if (!SPARSE && p.masks_out) {                             // the union over the tokens of !(result < threshold), one bit per row
                for (int k0 = warp * 32; k0 < n_tile; k0 += MM_WARPS * 32) {
                    const int k = k0 + lane;
                    bool any = false;
                    for (int t = 0; t < p.T && k < n_tile; t++) {
                        float o = sum_of(k, t);
                        if (p.bias) o += p.bias[lo + first + k];
                        if (p.relu) o = fmaxf(o, 0.f);
                        any |= !(o < p.masks_threshold);
                    }
                    const uint32_t m = __ballot_sync(0xffffffffu, any);
                    if (lane < 4 && k0 + lane * 8 < n_tile) {         // the range starts at a multiple of 8 rows
                        unsigned char * o = reinterpret_cast<unsigned char *>(p.masks_out) + (lo + first + k0) / 8 + lane;
                        const unsigned char bits = (unsigned char)(m >> (lane * 8));
                        *o = p.masks_or ? (unsigned char)(*o | bits) : bits;
                    }
                }
            }
            clear();
        }
        if (++slice == p.n_slices) { slice = 0; tile++; }
    }
}

// ---------------------------------------------------------------------------------------------- launch
template <int WT, int NT, int TM, bool SPARSE, bool GATED>
static int mm_go(MmP p, bool pdl, cudaStream_t st) {
    using Z = MmShape<WT, NT, TM>;
    p.n_slices = (p.ncols + Z::KS - 1) / Z::KS;
    // (8 rows are as little as is worth a CTA: its share of the activation costs more than its weights)
    const int G = (int)imin64(sm_count(), (p.nrows + 7) / 8);
    p.max_rows = SPARSE ? (p.nrows + G - 1) / G + 1 : 0;
    if (p.max_rows * 4 > 8192 - 256) return PI_ERR_UNSUPPORTED;       // (more than MM_MAX_ROWS rows)
    const size_t smem = Z::RED + (size_t)Z::S * Z::STAGE + (size_t)p.max_rows * 4;
    static bool attr_done[16] = {false};
    int dev = 0;
    PI_CUDA(cudaGetDevice(&dev));
    auto kern = k_mm<WT, NT, TM, SPARSE, GATED>;
    if (dev >= 0 && dev < 16 && !attr_done[dev]) {
        PI_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MM_SMEM_MAX));
        attr_done[dev] = true;
    }
    PI_CUDA(launch_k(kern, dim3(G), dim3(MM_THREADS), smem, st, pdl, p));
    return PI_OK;
}

template <int WT, int NT, int TM>
static int mm_sel(const MmP & p, bool pdl, cudaStream_t st) {
    if (!p.masks) return mm_go<WT, NT, TM, false, false>(p, pdl, st);
    if (p.W2)     return mm_go<WT, NT, TM, true, true>(p, pdl, st);
    return mm_go<WT, NT, TM, true, false>(p, pdl, st);
}

template <int WT, int NT>
static int mm_tile(const MmP & p, bool pdl, cudaStream_t st) {
    // the smallest tile that holds a CTA's share of the rows: less column splitting inside the CTA for the taller ones
    const int64_t share = ((int64_t)p.nrows * (p.W2 ? 2 : 1) + sm_count() - 1) / sm_count();
    if (share > 64) return mm_sel<WT, NT, 128>(p, pdl, st);
    if (share > 32) return mm_sel<WT, NT, 64>(p, pdl, st);
    return mm_sel<WT, NT, 32>(p, pdl, st);
}

// PI_ERR_UNSUPPORTED: shape not eligible, the caller uses another kernel.  Tokens go in launches of at most 32.
int launch_mm(const GemvArgs & a, cudaStream_t st) {
    const bool q4 = a.wtype == PI_TYPE_Q4_0;
    if (q4 ? !a.x.lo || a.ncols % 256 != 0 : !a.x.h16 || a.ncols % 8 != 0) return PI_ERR_UNSUPPORTED;
    if (a.nrows > (a.masks ? MM_MAX_ROWS : (1 << 26)) || (a.W2 && !a.masks) || (a.list && !a.masks)) return PI_ERR_UNSUPPORTED;
    for (int t0 = 0; t0 < a.T; t0 += 32) {
        MmP p;
        p.W = (const uint8_t *)a.W; p.W2 = (const uint8_t *)a.W2; p.row_bytes = (int64_t)pi_row_bytes(a.wtype, a.ncols);
        p.nrows = (int)a.nrows; p.ncols = (int)a.ncols; p.nb = (int)(a.ncols / 32);
        p.T = a.T - t0 < 32 ? a.T - t0 : 32;
        if (q4) {
            p.x.lo = a.x.lo + (size_t)t0 * p.nb; p.x.hi = a.x.hi + (size_t)t0 * p.nb; p.x.d = a.x.d + (size_t)t0 * p.nb;
        } else {
            p.x.h16 = a.x.h16 + (size_t)t0 * a.ncols;
        }
        p.masks = a.masks; p.bucket = a.bucket; p.list = a.list_out; p.count = a.count_out; p.rows_total = t0 == 0 ? a.rows_total : nullptr;
        p.idx = a.idx ? a.idx + (size_t)t0 * a.idx_stride : nullptr; p.idx_stride = a.idx_stride; p.threshold = a.threshold;
        p.bias = a.bias; p.relu = a.relu;
        p.dst = a.dst ? a.dst + (size_t)t0 * a.dst_stride : nullptr;
        p.dst16 = a.dst16 ? a.dst16 + (size_t)t0 * a.dst_stride : nullptr; p.dst_stride = a.dst_stride;
        p.coef = a.coef ? a.coef + (size_t)t0 * a.coef_stride : nullptr; p.coef_stride = a.coef_stride;
        p.masks_out = a.masks_out; p.masks_threshold = a.masks_threshold; p.masks_or = t0 > 0;
        p.n_slices = 0; p.max_rows = 0;
        int rc;
        if (q4) rc = p.T <= 8 ? mm_tile<PI_TYPE_Q4_0, 1>(p, a.pdl, st) : p.T <= 16 ? mm_tile<PI_TYPE_Q4_0, 2>(p, a.pdl, st) : mm_tile<PI_TYPE_Q4_0, 4>(p, a.pdl, st);
        else    rc = p.T <= 8 ? mm_tile<PI_TYPE_F16, 1>(p, a.pdl, st) : p.T <= 16 ? mm_tile<PI_TYPE_F16, 2>(p, a.pdl, st) : mm_tile<PI_TYPE_F16, 4>(p, a.pdl, st);
        if (rc != PI_OK) return rc;
    }
    return PI_OK;
}

}  // namespace pi
