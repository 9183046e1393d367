// ggml_axpy for many tokens on tcgen05: dst[t, c] = sum over listed rows r of coef[t, r] * Wt[r, c], coefficients and (dequantised) weights as
// halves, FP32 sums: what pi_axpy_mm.cu computes for FP16 rows, and for Q4_0 rows whose factors are rounded to FP16 (exact factors stay there).
//
// Bound: with 256 tokens the coefficients that an SM brings in (2.6 MB of 5160 list positions) and the products (44 us of 28672 x 8192, 72 %), with
// fewer the rows.  mma.sync read every fragment of both operands through registers and expanded the nibbles once per 64 tokens.
//
// As a product D[t, c] += A[t, r] * B[r, c]: tokens are the 128 lanes (M; two tiles beyond 128), CW columns the columns (N), list positions K.
// The rows lie in memory with c contiguous, so B is MN-major: a row's 128-byte piece of 64 columns is a row of the swizzled operand as
// it is.  Sums stay in tensor memory for a CTA's whole range of list positions, in as many accumulators as it has room for (512 columns), one
// stage each in turn: the tensor cores cut FP32 sums at every step, so that the error grows with the length of a chain (one accumulator
// for 128 tokens and 4096 columns 1.07e-6 of the result, two 0.53e-6; mma.sync 0.98e-6).
//
// Work split: a CTA has CW columns, all tokens and one of `split` equal ranges of the list (steps of 64); it writes one partial vector, which the
// next norm adds.  256 columns where that leaves at least 8 ranges of columns: the coefficients are read once per range.  At most 16
// partial vectors: more would cost their reader more than they save.
//
// Warps: 0 brings the coefficients as TMA tiles (by list position; zeros behind the last one, which their writer leaves there), 1 issues
// the products, 2..15 bring the rows through registers, nibbles expanded on the way, and 4..15 write the sums.  Rows come in tasks of 2 KB
// (Q4_0: 64 blocks), 16 (8) a stage of 256 columns, dealt to the warps in turn, the next two on their way while one is stored.
//
// us, mma.sync | here: 28672 x 8192 Q4_0, 78 % of the rows, 256 tokens 375 | 104 (470 MB through L2 in 80 us: every range of columns reads all
// coefficients); 11008 x 4096 FP16, 72 %, 77 tokens 38 | 24; 75 %, as operators with 12 us of
// preparation and sum, 77 tokens 52 | 33, 128 79 | 39, 256 138 | 66.
#include "pi_tc.cuh"

namespace pi {

static constexpr int XT_THREADS = 512, XT_SMAX = 6, XT_KS = 64;       // stages at most; list positions of a stage
static constexpr int XT_SMEM_MAX = 226 * 1024, XT_RING = XT_SMEM_MAX - 1024;

struct alignas(64) XtP {
    CUtensorMap m_c;
    const uint8_t * Wt; int64_t row_bytes; int nrows, ncols, nb;
    int T, nt, c_rows;                                                // token tiles (1, 2), rows of a coefficient box
    const int32_t * list; const int32_t * count;
    float * partial; int64_t piece; int split;                        // floats between partial vectors
    unsigned int * status;
};

__device__ __forceinline__ uint32_t xt_mul2(uint32_t a, uint32_t b) { uint32_t r; asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ uint32_t xt_add2(uint32_t a, uint32_t b) { uint32_t r; asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ uint32_t xt_fma2(uint32_t a, uint32_t b, uint32_t c) { uint32_t r; asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c)); return r; }

template <bool Q4, int CW>
__global__ void __launch_bounds__(XT_THREADS, 1) k_axpy_tc(const __grid_constant__ XtP p) {
    constexpr int TASKS = Q4 && CW == 256 ? 8 : CW / 16, NW = 14;                           // tasks of a stage; warps that bring rows
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ uint64_t s_full[XT_SMAX], s_empty[XT_SMAX], s_done;
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_dead;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);    // (uniform for the compiler)
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int range = blockIdx.x / p.split, mine = blockIdx.x % p.split, col0 = range * CW;
    if (tid < XT_SMAX) { mbar_init(s_full + tid, 1 + TASKS); mbar_init(s_empty + tid, 1); }
    if (tid == 0) { mbar_init(&s_done, 1); s_dead = 0; }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (warp == 0) tc_alloc(&s_tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem, 0);
    pdl_launch();
    auto wait = [&](uint64_t * bar, unsigned parity) -> bool {        // warp-uniform; false: the wait ran out, here or elsewhere
        bool ok = false;
        for (int spins = 0; spins < (1 << 20) && !ok && !s_dead; spins++) ok = mbar_try_wait(bar, parity);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok && lane == 0) { s_dead = 1; if (p.status) atomicOr(p.status, 16u); }
        return ok;
    };
    pdl_wait();
    const int n = __shfl_sync(0xffffffffu, min(*p.count, p.nrows), 0), all = (n + XT_KS - 1) / XT_KS;
    const int st0 = (int)((long long)all * mine / p.split), n_st = (int)((long long)all * (mine + 1) / p.split) - st0;      // my stages of the list
    const uint32_t w_off = p.nt > 1 ? 32768u : (uint32_t)p.c_rows * 128u, stage = w_off + (uint32_t)CW * 128u;
    const int S = min(XT_SMAX, XT_RING / (int)stage), accs = 512 / (p.nt * CW);

    if (warp == 0) {
        // ================================================================= coefficients
        int slot = 0;
        unsigned phase = 1u;                                          // parity of the hand-back to wait for (first round: none)
        int i = 0;
        for (; i < n_st; i++) {
            if (!wait(s_empty + slot, phase)) break;
            if (lane == 0) {
                mbar_expect_tx(s_full + slot, (unsigned)(p.nt * p.c_rows * 128));
                for (int t = 0; t < p.nt; t++) tma_tile(ring + (uint32_t)slot * stage + t * 16384, &p.m_c, (st0 + i) * XT_KS, t * 128, s_full + slot);
            }
            __syncwarp();
            if (++slot == S) { slot = 0; phase ^= 1u; }
        }
        if (lane == 0) ring_land(s_full, i, S);
        __syncwarp();
    } else if (warp == 1) {
        // ================================================================= products
        constexpr uint32_t idesc = tc_idesc(CW, true);
        int slot = 0, acc = 0;
        unsigned phase = 0u;
        for (int i = 0; i < n_st; i++) {
            if (!wait(s_full + slot, phase)) break;
            tc_fence_after();
            const uint32_t base = ring + (uint32_t)slot * stage;
            const uint64_t a = tc_desc_k(base), w = tc_desc_mn(base + w_off, XT_KS * 128);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t d = tmem + (uint32_t)(acc * p.nt * CW);
                tc_mma_f16(d, a + 2 * k, w + 128 * k, idesc, i >= accs || k > 0);
                if (p.nt > 1) tc_mma_f16(d + CW, a + 1024 + 2 * k, w + 128 * k, idesc, i >= accs || k > 0);
            }
            if (++acc == accs) acc = 0;
            tc_commit(s_empty + slot);
            if (++slot == S) { slot = 0; phase ^= 1u; }
        }
        tc_commit(&s_done);                                           // nothing is in flight when tensor memory is given back
        for (int spins = 0; spins < (1 << 20) && !mbar_try_wait(&s_done, 0u); spins++) {}
        __syncwarp();
    } else {
        // ================================================================= rows
        const int pw = warp - 2, n_tasks = n_st * TASKS;
        int slot = 0, at_stage = 0;
        unsigned phase = 1u;
        bool ok = true;
        auto take_slot = [&](int stage_no) -> uint32_t {              // address of the rows in the stage's slot, free
            for (; at_stage < stage_no; at_stage++)
                if (++slot == S) { slot = 0; phase ^= 1u; }
            ok = wait(s_empty + slot, phase) && ok;
            return ring + (uint32_t)slot * stage + w_off;
        };
        auto hand_over = [&]() {
            tc_fence_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(s_full + slot);
        };
        auto entry = [&](int task, int r) -> int { return (st0 + task / TASKS) * XT_KS + r; };        // of the list: entry r of the task's stage
        if (!Q4) {
            // 16 bytes a lane, LPR lanes a row, four rows a lane
            constexpr int LPR = CW / 8, RPI = 32 / LPR, RT = XT_KS / TASKS;
            const int piece = lane % LPR, r0 = lane / LPR, col = col0 + piece * 8;
            const bool in = col < p.ncols;
            int row[4];
            uint4 v[3][4];
            auto numbers = [&](int task) {                            // row numbers, < 0 where there is none
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int at = entry(task, task % TASKS * RT + r0 + j * RPI), v = task < n_tasks && at < n ? p.list[at] : -1;
                    row[j] = v < p.nrows ? v : -1;
                }
            };
            auto load = [&](int task, uint4 (&b)[4]) {
#pragma unroll
                for (int j = 0; j < 4; j++) b[j] = in && row[j] >= 0 ? ldg_stream(p.Wt + (size_t)row[j] * p.row_bytes + (size_t)col * 2) : make_uint4(0u, 0u, 0u, 0u);
                numbers(task + NW);
            };
            auto store = [&](int task, const uint4 (&b)[4]) {
                if (task >= n_tasks) return;
                const uint32_t at = take_slot(task / TASKS) + (uint32_t)(piece >> 3) * (XT_KS * 128);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int r = task % TASKS * RT + r0 + j * RPI;
                    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" :: "r"(at + (uint32_t)(r * 128 + ((piece ^ r) & 7) * 16)), "r"(b[j].x), "r"(b[j].y), "r"(b[j].z), "r"(b[j].w) : "memory");
                }
                hand_over();
            };
            numbers(pw);
            load(pw, v[0]);
            load(pw + NW, v[1]);
            for (int g = pw; g < n_tasks && ok; g += 3 * NW) {
                load(g + 2 * NW, v[2]); store(g, v[0]);
                load(g + 3 * NW, v[0]); store(g + NW, v[1]);
                load(g + 4 * NW, v[1]); store(g + 2 * NW, v[2]);
            }
        } else {
            // NU blocks (16 bytes of nibbles and a scale) a lane: 8 rows x 8 (4) blocks, so that the lanes that store together have 8 different rows and
            // with them different banks
            constexpr int NU = CW >= 256 ? 2 : 1, RT = XT_KS / TASKS;
            const int r0 = lane & 7, b0 = lane >> 3;
            // (nothing looks at what is loaded before the next task's turn: the row number's validity follows from its place)
            auto number = [&](int task, int r) -> int { return __ldg(p.list + max(0, min(entry(task, r), n - 1))); };
            auto start_of = [&](int v) -> const uint8_t * { return p.Wt + (size_t)min((unsigned)v, (unsigned)(p.nrows - 1)) * p.row_bytes; };
            int row = number(pw, pw % TASKS * RT + r0);
            uint4 q[3][NU];
            unsigned short s[3][NU];
            auto load = [&](int task, uint4 (&b)[NU], unsigned short (&d)[NU]) {
                const uint8_t * src = start_of(row) + (size_t)(col0 / 32 + b0) * 16, * scale = start_of(row) + (size_t)p.nb * 16 + (size_t)(col0 / 32 + b0) * 2;
#pragma unroll
                for (int j = 0; j < NU; j++) {
                    b[j] = ldg_stream(src + j * 64);
                    d[j] = __ldg(reinterpret_cast<const unsigned short *>(scale + j * 8));
                }
                row = number(task + NW, (task + NW) % TASKS * RT + r0);
            };
            auto store = [&](int task, const uint4 (&b)[NU], const unsigned short (&d)[NU]) {
                if (task >= n_tasks) return;
                const int r = task % TASKS * RT + r0;
                const bool is = entry(task, r) < n;
                uint32_t o[NU][4][4];                                 // 8 columns each: low nibbles of bytes 0..7, 8..15, then the high ones
#pragma unroll
                for (int j = 0; j < NU; j++) {
                    const uint32_t sc = is ? (uint32_t)d[j] * 0x10001u : 0u;         // (no row: weights of 0)
                    const uint32_t w[4] = {b[j].x, b[j].y, b[j].z, b[j].w};
#pragma unroll
                    for (int k = 0; k < 4; k++) {                     // (bit patterns: 0x6400 = 1024, 0x2C00 = 1/16, 0xE408 = -1032, 0xD480 = -72)
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const uint32_t x = __byte_perm(w[k], 0u, h ? 0x4342 : 0x4140);
                            o[j][k >> 1][(k & 1) * 2 + h] = xt_mul2(xt_add2((x & 0x000F000Fu) | 0x64006400u, 0xE408E408u), sc);
                            o[j][2 + (k >> 1)][(k & 1) * 2 + h] = xt_mul2(xt_fma2((x & 0x00F000F0u) | 0x64006400u, 0x2C002C00u, 0xD480D480u), sc);
                        }
                    }
                }
                const uint32_t at = take_slot(task / TASKS) + (uint32_t)(r * 128);
#pragma unroll
                for (int j = 0; j < NU; j++) {
                    const int blk = b0 + 4 * j;
                    const uint32_t to = at + (uint32_t)(blk >> 1) * (XT_KS * 128);
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" :: "r"(to + (uint32_t)((((blk & 1) * 4 + c) ^ (r & 7)) * 16)), "r"(o[j][c][0]), "r"(o[j][c][1]), "r"(o[j][c][2]), "r"(o[j][c][3]) : "memory");
                }
                hand_over();
            };
            load(pw, q[0], s[0]);
            load(pw + NW, q[1], s[1]);
            for (int g = pw; g < n_tasks && ok; g += 3 * NW) {
                load(g + 2 * NW, q[2], s[2]); store(g, q[0], s[0]);
                load(g + 3 * NW, q[0], s[0]); store(g + NW, q[1], s[1]);
                load(g + 4 * NW, q[1], s[1]); store(g + 2 * NW, q[2], s[2]);
            }
        }
        // ================================================================= sums: a thread has one token's columns
        // Four lanes store 64 bytes of a token, through the ring, which is free (a lane its own token's 16 bytes at a time: 13824 x 5120, 256 tokens, 3 % of
        // the rows, 63 us where mma.sync takes 58; so 53; 75 % 92 -> 83)
        if (warp >= 4) wait(&s_done, 0u);
        float * const turn = reinterpret_cast<float *>(smem_raw + (ring - smem_u32(smem_raw))) + (warp - 4) * (32 * 20);
        tc_fence_after();
        for (int t = 0; t < p.nt && warp >= 4; t++) {
            const int tok0 = t * 128 + (warp & 3) * 32;
            if (tok0 >= p.T) break;
            for (int c = ((warp >> 2) - 1) * 16; c < CW; c += 48) {
                if (col0 + c >= p.ncols) break;
                float v[16];
#pragma unroll
                for (int j = 0; j < 16; j++) v[j] = 0.f;              // (no row in my range)
                for (int k = 0; k < min(accs, n_st); k++) {
                    float w[16];
                    tc_ld16(w, tmem + (uint32_t)((warp & 3) * 32 << 16) + (uint32_t)((k * p.nt + t) * CW + c));
#pragma unroll
                    for (int j = 0; j < 16; j++) v[j] += w[j];
                }
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4 *>(turn + lane * 20 + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                __syncwarp();
                const int part = (lane & 3) * 4;
                float * o = p.partial + (size_t)mine * p.piece + (size_t)(tok0 + (lane >> 2)) * p.ncols + col0 + c + part;
#pragma unroll
                for (int j = 0; j < 32; j += 8, o += 8 * (size_t)p.ncols)           // (a multiple of 8 columns)
                    if (tok0 + j + (lane >> 2) < p.T && col0 + c + part < p.ncols) *reinterpret_cast<float4 *>(o) = *reinterpret_cast<const float4 *>(turn + (j + (lane >> 2)) * 20 + part);
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tc_dealloc(tmem, 512);
}

// ---------------------------------------------------------------------------------------------- launch
static int xt_columns(int64_t ncols) { return ncols >= 2048 ? 256 : ncols >= 1024 ? 128 : 64; }

int axpy_tc_pieces(int64_t ncols) {
    const int64_t ranges = (ncols + xt_columns(ncols) - 1) / xt_columns(ncols), s = sm_count() / ranges;
    return s < 1 ? 1 : s > 16 ? 16 : (int)s;
}

template <bool Q4, int CW>
static int xt_go(const XtP & p, bool pdl, cudaStream_t st) {
    static bool attr_done[16] = {false};
    int dev = 0;
    PI_CUDA(cudaGetDevice(&dev));
    auto kern = k_axpy_tc<Q4, CW>;
    if (dev >= 0 && dev < 16 && !attr_done[dev]) {
        PI_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, XT_SMEM_MAX));
        attr_done[dev] = true;
    }
    PI_CUDA(launch_k(kern, dim3((p.ncols + CW - 1) / CW * p.split), dim3(XT_THREADS), (size_t)XT_SMEM_MAX, st, pdl, p));
    return PI_OK;
}

// Called by launch_axpy_mm, which has checked the arguments and the room for axpy_tc_pieces partial vectors.  Tokens go in launches of at most 256.
int launch_axpy_tc(const AxpyArgs & a, cudaStream_t st, int * pieces_used) {
    const int split = axpy_tc_pieces(a.ncols), cw = xt_columns(a.ncols);
    if (pieces_used) *pieces_used = split;
    for (int t0 = 0; t0 < a.T; t0 += 256) {
        XtP p;
        p.T = a.T - t0 < 256 ? a.T - t0 : 256;
        p.nt = (p.T + 127) / 128; p.c_rows = p.nt > 1 ? 128 : (p.T + 7) / 8 * 8;
        int rc = tensor_map(&p.m_c, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, (const __half *)a.coef + (size_t)t0 * a.coef_stride, a.coef_stride, p.T, a.coef_stride * 2, XT_KS, p.c_rows, CU_TENSOR_MAP_SWIZZLE_128B);
        if (rc != PI_OK) return rc;
        p.Wt = (const uint8_t *)a.Wt; p.row_bytes = (int64_t)pi_row_bytes(a.wtype, a.ncols); p.nrows = (int)a.nrows; p.ncols = (int)a.ncols; p.nb = (int)(a.ncols / 32);
        p.list = a.list; p.count = a.count; p.status = a.status;
        p.partial = a.partial + (size_t)t0 * a.ncols; p.piece = (int64_t)a.T * a.ncols; p.split = split;
        const bool q4 = a.wtype == PI_TYPE_Q4_0;
        rc = cw == 256 ? (q4 ? xt_go<true, 256>(p, a.pdl, st) : xt_go<false, 256>(p, a.pdl, st))
           : cw == 128 ? (q4 ? xt_go<true, 128>(p, a.pdl, st) : xt_go<false, 128>(p, a.pdl, st))
                       : q4 ? PI_ERR_UNSUPPORTED : xt_go<false, 64>(p, a.pdl, st);          // (rounded Q4_0 factors: whole 1024 columns)
        if (rc != PI_OK) return rc;
    }
    return PI_OK;
}

}  // namespace pi
