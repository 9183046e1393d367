// llm_build_kv_store + llm_build_kqv (llama.cpp:4383-4418, 4764-4850) for several tokens of a step, on the tensor cores.
//
// A CTA takes 16 query rows that read the same keys and values: the query heads that share a KV head, of one token (a batch of
// sequences), or 16 consecutive tokens of one head (a prompt chunk).  The kernel with one CTA per (head, token) reads a KV
// head once for every query head and token and keeps one CTA per SM: 57 us for 32 sequences of 190 positions with 32 heads
// (92 MB of keys and values), 125 us for 32 prompt tokens with 64 heads.
//
// Bound: the bytes of the cached rows for batches, the chain scores -> maximum -> probabilities -> values for chunks.
// A probability takes the place of a score, and the output sums that of the values: what shared memory holds decides how many CTAs an SM has (256
// tokens with 64 heads in a context of 768: 113 KB and one CTA an SM before, 89 KB and two now, the longest ones first: 48 -> 45 us).
// Scores: mma.m16n8k16 with the keys straight from global memory: a lane loads 16 bytes (8 columns) of a row, which serve
// as B operands of two mma whose k order is permuted in the same way on the query side; four tiles of 8 positions in
// flight per warp, or two where more than two CTAs per SM have work (attn_mm_go).  Values travel to shared memory by cp.async (tiles of 64 positions, two in flight) while the scores are made and
// are read transposed.  Every CTA rotates and stores the new keys and values it reads itself (CTAs that share a KV head store the
// same bits), so no store pass runs before a chunk of up to AM_OWN_STORE tokens; beyond that the repeated work costs more than a launch.
// Numerics follow the CPU path as in k_attention: q, k, v and the probabilities in FP16, exp through FP16, the normaliser
// summed in double.
#include "pi_act.cuh"

namespace pi {

static constexpr int AM_THREADS = 256, AM_WARPS = 8, AM_VT = 64;      // positions of a value tile
static constexpr int AM_OWN_STORE = 32;

struct AttnMmP {
    const float * q; const float * k; const float * v; __half * k_cache; __half * v_cache;
    const int32_t * seq; const int32_t * pos; int T, n_head, n_head_kv, n_ctx;
    const float * cs; int neox; int64_t q_stride, kv_stride;
    float * out; ActBuf out_act; int out_act_type;
    int chunk;                                                        // rows are tokens of one head, else heads of one token
    int stored;                                                       // the new keys and values are in the cache already
    int P, R;                                                         // positions (a multiple of 64) and rows that shared memory holds
};

__device__ __forceinline__ void am_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int HC, int UN>                                             // head_dim / 32; tiles of 8 positions in flight per warp
__global__ void __launch_bounds__(AM_THREADS, UN == 2 ? 4 : HC == 2 ? 3 : 2) k_attention_mm(const AttnMmP p) {
    constexpr int HD = HC * 32, HALF = HD / 2;
    constexpr int V_PITCH = HD + 8, Q_PITCH = HD + 8;                 // halves; odd multiples of 16 bytes
    constexpr int NWC = HD / 16 < AM_WARPS ? HD / 16 : AM_WARPS;      // warps along the value columns, the rest split the positions
    constexpr int KSPL = AM_WARPS / NWC, NCG = HD / 16 / NWC;         // column groups of 16 per warp
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_pos[16];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
    const int group = p.n_head / p.n_head_kv, dkv = p.n_head_kv * HD;
    // shared-memory map: scores [R][P + 4] F32, later the probabilities as FP16 in their place | queries [16][Q_PITCH] | values 2 x [64][V_PITCH], later the output sums
    const int S_PITCH = p.P + 4, P_PITCH = 2 * S_PITCH;
    float * sc = reinterpret_cast<float *>(smem);
    __half * p16 = reinterpret_cast<__half *>(smem);
    __half * qs = reinterpret_cast<__half *>(smem + ((size_t)p.R * S_PITCH * 4 + 127) / 128 * 128);
    __half * vs = qs + 16 * Q_PITCH;

    pdl_launch();
    // ---- before the wait: positions, and L2 hints for the cached rows (earlier steps wrote them)
    int t0, n_rows, head0, hk;
    if (p.chunk) {
        head0 = blockIdx.x; hk = head0 / group; t0 = (gridDim.y - 1 - blockIdx.y) * 16; n_rows = min(16, p.T - t0);
    } else {
        const int ng = (group + 15) / 16, gi = blockIdx.x % ng;
        hk = blockIdx.x / ng; head0 = hk * group + gi * 16; t0 = blockIdx.y; n_rows = min(16, group - gi * 16);
    }
    const int sq = p.seq ? p.seq[t0] : 0;
    __half * kc = p.k_cache + ((size_t)sq * p.n_ctx * p.n_head_kv + hk) * HD;
    __half * vc = p.v_cache + ((size_t)sq * p.n_ctx * p.n_head_kv + hk) * HD;
    // tokens whose new keys and values this CTA stores: its own, or all of the chunk up to its last
    const int s_lo = p.chunk ? 0 : t0, s_n = p.stored ? 0 : p.chunk ? t0 + n_rows : 1;
    int n_keys = 0;                                                   // keys that any row sees
    for (int r = 0; r < (p.chunk ? n_rows : 1); r++) { const int ps = p.pos[t0 + r]; if (ps >= 0 && ps < p.n_ctx) n_keys = max(n_keys, ps + 1); }
    if (n_keys == 0) return;                                          // never index the cache out of range
    if (tid < 16) {
        const int ps = tid < n_rows ? p.pos[p.chunk ? t0 + tid : t0] : -1;
        s_pos[tid] = ps < p.n_ctx ? ps : -1;
    }
    for (int j = tid; j < n_keys; j += AM_THREADS) {
        const char * kr = reinterpret_cast<const char *>(kc + (size_t)j * dkv), * vr = reinterpret_cast<const char *>(vc + (size_t)j * dkv);
#pragma unroll
        for (int o = 0; o < HD * 2; o += 128) {
            asm volatile("prefetch.global.L2 [%0];" :: "l"(kr + o));
            asm volatile("prefetch.global.L2 [%0];" :: "l"(vr + o));
        }
    }
    pdl_wait();

    // ---- queries (rotated, FP16) to shared memory; the new keys and values to the cache
    // (every load first, the first new key and value included, so that their latencies pass together: eight layers of 32 sequences
    // 1237 -> 1224 us per pass, three layers of 8 sequences with 8 KV heads 544 -> 540 us, softmax loops in steps of four included)
    constexpr int QI = 16 * HALF / AM_THREADS;
    float q0[QI], q1[QI]; float2 qr[QI];
    const bool pairs = p.cs && !p.neox;                               // rotated pairs are neighbours, else a half apart
#pragma unroll
    for (int i = 0; i < QI; i++) {
        const int e = tid + i * AM_THREADS, r = e / HALF, k = e % HALF, t = p.chunk ? t0 + r : t0;
        q0[i] = q1[i] = 0.f; qr[i] = make_float2(1.f, 0.f);
        if (r < n_rows) {
            const float * qh = p.q + (size_t)t * p.q_stride + (size_t)(p.chunk ? head0 : head0 + r) * HD;
            q0[i] = qh[pairs ? 2 * k : k]; q1[i] = qh[pairs ? 2 * k + 1 : k + HALF];
            const int ps = p.pos[t];
            if (p.cs && ps >= 0 && ps < p.n_ctx) qr[i] = reinterpret_cast<const float2 *>(p.cs)[(size_t)ps * HALF + k];
        }
    }
    int n_ps = -1; float n_k0 = 0.f, n_k1 = 0.f, n_v0 = 0.f, n_v1 = 0.f; float2 n_r = make_float2(1.f, 0.f);
    auto load_new = [&](int e) {
        n_ps = -1;
        if (e >= s_n * HALF) return;
        const int t = s_lo + e / HALF, k = e % HALF, ps = p.pos[t];
        if (ps < 0 || ps >= p.n_ctx) return;
        const float * kh = p.k + (size_t)t * p.kv_stride + (size_t)hk * HD, * vh = p.v + (size_t)t * p.kv_stride + (size_t)hk * HD;
        n_ps = ps; n_k0 = kh[pairs ? 2 * k : k]; n_k1 = kh[pairs ? 2 * k + 1 : k + HALF]; n_v0 = vh[k]; n_v1 = vh[k + HALF];
        if (p.cs) n_r = reinterpret_cast<const float2 *>(p.cs)[(size_t)ps * HALF + k];
    };
    load_new(tid);
#pragma unroll
    for (int i = 0; i < QI; i++) {
        const int e = tid + i * AM_THREADS, r = e / HALF, k = e % HALF;
        float o0 = q0[i], o1 = q1[i];
        if (p.cs) rope_pair(q0[i], q1[i], qr[i].x, qr[i].y, o0, o1);
        qs[r * Q_PITCH + (pairs ? 2 * k : k)] = __float2half_rn(o0);
        qs[r * Q_PITCH + (pairs ? 2 * k + 1 : k + HALF)] = __float2half_rn(o1);
    }
    for (int e = tid; e < s_n * HALF; e += AM_THREADS) {
        const int k = e % HALF, ps = n_ps;
        float o0 = n_k0, o1 = n_k1;
        const float v0 = n_v0, v1 = n_v1;
        if (p.cs) rope_pair(n_k0, n_k1, n_r.x, n_r.y, o0, o1);
        load_new(e + AM_THREADS);
        if (ps < 0) continue;
        kc[(size_t)ps * dkv + (pairs ? 2 * k : k)] = __float2half_rn(o0);
        kc[(size_t)ps * dkv + (pairs ? 2 * k + 1 : k + HALF)] = __float2half_rn(o1);
        vc[(size_t)ps * dkv + k] = __float2half_rn(v0);
        vc[(size_t)ps * dkv + k + HALF] = __float2half_rn(v1);
    }
    __syncthreads();                                                  // this CTA's stores are visible to all of its threads

    auto issue_v = [&](int tile) {
        const uint32_t base = smem_u32(vs + (size_t)(tile & 1) * AM_VT * V_PITCH);
        for (int e = tid; e < AM_VT * (HD / 8); e += AM_THREADS) {
            const int r = e / (HD / 8), c = e % (HD / 8), j = tile * AM_VT + r;
            const bool in = j < n_keys;                               // rows past the last key: zeros (their probabilities are 0)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(base + (uint32_t)(r * V_PITCH + c * 8) * 2), "l"(vc + (size_t)(in ? j : 0) * dkv + c * 8), "r"(in ? 16u : 0u) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int n_vt = (n_keys + AM_VT - 1) / AM_VT;
    issue_v(0);
    if (n_vt > 1) issue_v(1);

    // ---- scores
    {
        uint32_t aq[HC][2][4];                                        // 8 columns of rows g and g + 8 per 32
#pragma unroll
        for (int c = 0; c < HC; c++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint4 v = *reinterpret_cast<const uint4 *>(qs + (g + 8 * h) * Q_PITCH + c * 32 + q * 8);
                aq[c][h][0] = v.x; aq[c][h][1] = v.y; aq[c][h][2] = v.z; aq[c][h][3] = v.w;
            }
        const float scale = 1.0f / sqrtf((float)HD);
        const int n_tiles = (n_keys + 7) / 8;
        for (int nt0 = warp; nt0 < n_tiles; nt0 += AM_WARPS * UN) {
            uint4 kv[UN][HC];
#pragma unroll
            for (int u = 0; u < UN; u++) {
                const int j = min((nt0 + u * AM_WARPS) * 8 + g, n_keys - 1);
#pragma unroll
                for (int c = 0; c < HC; c++) kv[u][c] = __ldcg(reinterpret_cast<const uint4 *>(kc + (size_t)j * dkv + c * 32 + q * 8));
            }
#pragma unroll
            for (int u = 0; u < UN; u++) {
                const int nt = nt0 + u * AM_WARPS;
                if (nt >= n_tiles) break;
                float c4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int c = 0; c < HC; c++) {
                    am_mma(c4, aq[c][0][0], aq[c][1][0], aq[c][0][1], aq[c][1][1], kv[u][c].x, kv[u][c].y);
                    am_mma(c4, aq[c][0][2], aq[c][1][2], aq[c][0][3], aq[c][1][3], kv[u][c].z, kv[u][c].w);
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int r = g + 8 * h, j = nt * 8 + 2 * q;
                    if (r >= p.R) continue;
                    const int last = s_pos[r];
                    sc[r * S_PITCH + j]     = j     <= last ? c4[2 * h] * scale     : -INFINITY;
                    sc[r * S_PITCH + j + 1] = j + 1 <= last ? c4[2 * h + 1] * scale : -INFINITY;
                }
            }
        }
    }
    __syncthreads();

    // ---- softmax (ggml.c:10708-10777), a warp per row
    const int k_end = (n_keys + 15) / 16 * 16;
    for (int r = warp; r < p.R; r += AM_WARPS) {
        const int last = s_pos[r];
        float * row = sc + r * S_PITCH;
        float mx = -INFINITY;
#pragma unroll 4
        for (int j = lane; j <= last; j += 32) mx = fmaxf(mx, row[j]);
        mx = warp_max(mx);
        double part = 0.0;
#pragma unroll 4
        for (int j = lane; j <= last; j += 32) {
            const float e = round_f16(expf(round_f16(row[j] - mx)));
            row[j] = e;
            part += (double)e;
        }
        const float inv = (float)(1.0 / warp_sum_d(part));
        for (int j0 = lane; j0 < k_end + lane; j0 += 128) {            // (a probability takes the place of a score of its own step or an earlier one)
            float e[4];
#pragma unroll
            for (int u = 0; u < 4; u++) e[u] = j0 + 32 * u <= last ? row[j0 + 32 * u] * inv : 0.f;
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 4; u++) if (j0 + 32 * u < k_end) p16[r * P_PITCH + j0 + 32 * u] = __float2half_rn(e[u]);
        }
    }

    // ---- values
    float acc[NCG][2][4];
#pragma unroll
    for (int cg = 0; cg < NCG; cg++)
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[cg][m][j] = 0.f;
    const int wc = warp % NWC, wk = warp / NWC;
    const int r0 = min(g, p.R - 1), r1 = min(g + 8, p.R - 1);         // (fragment rows beyond R repeat the last one and are dropped)
    for (int tile = 0; tile < n_vt; tile++) {
        if (tile + 1 < n_vt) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else                 asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                              // the tile has landed for everybody (first time: the probabilities too)
        const uint32_t base = smem_u32(vs + (size_t)(tile & 1) * AM_VT * V_PITCH);
        for (int ks = wk; ks < AM_VT / 16; ks += KSPL) {
            const int j = tile * AM_VT + ks * 16;
            if (j >= k_end) break;
            const uint32_t a0 = *reinterpret_cast<const uint32_t *>(p16 + r0 * P_PITCH + j + 2 * q), a1 = *reinterpret_cast<const uint32_t *>(p16 + r1 * P_PITCH + j + 2 * q);
            const uint32_t a2 = *reinterpret_cast<const uint32_t *>(p16 + r0 * P_PITCH + j + 2 * q + 8), a3 = *reinterpret_cast<const uint32_t *>(p16 + r1 * P_PITCH + j + 2 * q + 8);
#pragma unroll
            for (int cg = 0; cg < NCG; cg++) {
                const int col = (cg * NWC + wc) * 16;
                uint32_t b[4];
                asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3])
                             : "r"(base + (uint32_t)((ks * 16 + (lane & 15)) * V_PITCH + col + (lane >> 4) * 8) * 2));
                am_mma(acc[cg][0], a0, a1, a2, a3, b[0], b[1]);
                am_mma(acc[cg][1], a0, a1, a2, a3, b[2], b[3]);
            }
        }
        if (tile + 2 < n_vt) { __syncthreads(); issue_v(tile + 2); }
    }
    // ---- the output rows (the values are dead: their place takes the sums of each position share)
    __syncthreads();
    float * o = reinterpret_cast<float *>(vs);
#pragma unroll
    for (int cg = 0; cg < NCG; cg++)
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int j = 0; j < 4; j++) o[(wk * 16 + g + (j >> 1) * 8) * HD + (cg * NWC + wc) * 16 + m * 8 + 2 * q + (j & 1)] = acc[cg][m][j];
    __syncthreads();
    for (int r = warp; r < n_rows; r += AM_WARPS) {
        if (s_pos[r] < 0) continue;
        const int t = p.chunk ? t0 + r : t0, h = p.chunk ? head0 : head0 + r;
        float y[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            y[j] = 0.f;
            if (lane < HD / 8) {
                y[j] = o[r * HD + lane * 8 + j];
                if (KSPL > 1) y[j] += o[(16 + r) * HD + lane * 8 + j];
                if (KSPL > 2) { y[j] += o[(32 + r) * HD + lane * 8 + j]; y[j] += o[(48 + r) * HD + lane * 8 + j]; }
            }
        }
        if (p.chunk) {
            // The rows of a chunk share their value tiles, so a row also multiplied the values of tokens after its own, by 0: one that is not
            // finite left a NaN.  Such a sum is made again from the row's own positions (and is a NaN if it is one).
            bool nan = false;
#pragma unroll
            for (int j = 0; j < 8; j++) nan |= y[j] != y[j];
            if (nan) {
#pragma unroll
                for (int j = 0; j < 8; j++) y[j] = 0.f;
                for (int i = 0; i <= s_pos[r]; i++) {
                    const float pi = __half2float(p16[r * P_PITCH + i]);
                    const uint4 w = __ldcg(reinterpret_cast<const uint4 *>(vc + (size_t)i * dkv) + lane);
                    const float2 w0 = h2f(w.x), w1 = h2f(w.y), w2 = h2f(w.z), w3 = h2f(w.w);
                    y[0] = fmaf(pi, w0.x, y[0]); y[1] = fmaf(pi, w0.y, y[1]); y[2] = fmaf(pi, w1.x, y[2]); y[3] = fmaf(pi, w1.y, y[3]);
                    y[4] = fmaf(pi, w2.x, y[4]); y[5] = fmaf(pi, w2.y, y[5]); y[6] = fmaf(pi, w3.x, y[6]); y[7] = fmaf(pi, w3.y, y[7]);
                }
            }
            __syncwarp();
        }
        if (p.out && lane < HD / 8) {                                 // (a caller's address: aligned to a float, not more)
            float * d = p.out + ((size_t)t * p.n_head + h) * HD + lane * 8;
#pragma unroll
            for (int j = 0; j < 8; j++) d[j] = y[j];
        }
        if (p.out_act_type) emit_act8(p.out_act_type, p.out_act, t, (int64_t)p.n_head * HD, h * (HD / 8) + lane, y, lane < HD / 8);
    }
}

// new keys (rotated) and values of a chunk's tokens to the cache: one thread per pair of columns
__global__ void __launch_bounds__(256) k_kv_store(const AttnMmP p, int hd) {
    const int half = hd / 2, e = blockIdx.x * 256 + threadIdx.x, t = blockIdx.y;
    pdl_launch();
    pdl_wait();
    if (e >= p.n_head_kv * half) return;
    const int hk = e / half, k = e % half, ps = p.pos[t];
    if (ps < 0 || ps >= p.n_ctx) return;
    const size_t row = (((size_t)(p.seq ? p.seq[t] : 0) * p.n_ctx + ps) * p.n_head_kv + hk) * hd;
    const float * kh = p.k + (size_t)t * p.kv_stride + (size_t)hk * hd, * vh = p.v + (size_t)t * p.kv_stride + (size_t)hk * hd;
    const int i0 = p.cs && !p.neox ? 2 * k : k, i1 = p.cs && !p.neox ? 2 * k + 1 : k + half;
    float o0 = kh[i0], o1 = kh[i1];
    if (p.cs) {
        const float2 a = reinterpret_cast<const float2 *>(p.cs)[(size_t)ps * half + k];
        rope_pair(kh[i0], kh[i1], a.x, a.y, o0, o1);
    }
    p.k_cache[row + i0] = __float2half_rn(o0);
    p.k_cache[row + i1] = __float2half_rn(o1);
    p.v_cache[row + k] = __float2half_rn(vh[k]);
    p.v_cache[row + k + half] = __float2half_rn(vh[k + half]);
}

static constexpr size_t AM_SMEM_MAX = 220 * 1024;

// rows and positions that shared memory holds, and its size
static size_t attn_mm_smem(const AttnArgs & a, int * P, int * R) {
    const int hd = a.head_dim, group = a.n_head / a.n_head_kv;
    *P = (a.n_ctx + 63) / 64 * 64;
    *R = a.store_mode != 0 || group > 16 ? 16 : group;
    auto up = [](size_t v) { return (v + 127) / 128 * 128; };
    return up((size_t)*R * (*P + 4) * 4) + (size_t)16 * (hd + 8) * 2 + (size_t)2 * AM_VT * (hd + 8) * 2;
}

// Several tokens and head_dim 64 or 128 whose scores fit; the others keep one CTA per head and token.  For prompt chunks of 32 tokens and more
// and at least 24 CTAs that is contexts of up to 2880 positions (256 tokens at the end of 2048, 32 heads of 128, 4 layers 4952 | 1276 us, of 2560
// 5611 | 1366; fewer CTAs leave the chip idle: at the end of 2560, 4 layers, 4 heads of 128 and 32 tokens, 8 CTAs, 296 | 417, 8 heads of 64 and
// 32 tokens, 16, 319 | 356; 40 tokens, 24, gain 4 .. 6 %, 16 heads of 64 and 32 tokens, 32, 14 .. 18 %); for the rest the line stays where
// scores and probabilities apart would fit (16 rows: about 1900 positions; 16 tokens at the end of 2304, 16 heads of 64, 314 | 346, of 2560, 32
// heads of 128 699 | 538).  So do steps of several sequences whose CTAs per head and token fit the SMs at once: nothing is gained there
// by reading a KV head once for all of its query heads, and a CTA of k_attention_row has more rows in flight.  us in k_attention_row | here,
// 8 sequences of 8 heads of 64: 200 positions 5.5 | 7.1, 1000 8.5 | 16.3, 3500 19.8 | 44.3; 4 of 32 heads of 128, 1000 positions
// 13.1 | 20.8.  With more CTAs than SMs: 32 sequences of 8 heads of 64 over 2 KV heads, 200 positions
// 9.6 | 7.1, 1000 15.8 | 16.4; 8 of 64 heads of 128 over 8 KV heads, 500 positions 28.0 | 13.2.
// Nor do steps with one or two query heads per KV head (one for 128) gain anything in long contexts: one or two rows of 16 are at work,
// and the scores take the room of what could be in flight.  16 sequences of 12 heads of 64, 4000 of 8192 positions 81.6 | 103.6, of 4096
// 81.0 | 75.9; 13 of 24 heads of 64 over 12 KV heads, 6000 of 8192 155.8 | 170.1; 13 of 12 heads of 128, 6000 of 12288 206 | 252, 32 of 32, 8000 of 8192
// 1050 | 1070.
bool attention_mm_takes(const AttnArgs & a) {
    int P, R;
    if (a.store_mode == 0 && (int64_t)a.T * a.n_head <= sm_count()) return false;
    if (a.store_mode == 0 && a.n_head / a.n_head_kv * a.head_dim <= 128 && a.n_ctx > 64 * a.head_dim) return false;
    if (!(a.T >= 2 && (a.head_dim == 64 || a.head_dim == 128) && a.n_ctx > 0)) return false;
    const size_t smem = attn_mm_smem(a, &P, &R);
    const bool many = a.store_mode != 0 && a.T >= 32 && (int64_t)a.n_head * ((a.T + 15) / 16) >= 24;
    return smem + (many ? 0 : (size_t)R * (P + 8) * 2) <= AM_SMEM_MAX;
}

// UN = 4 takes 126 registers with head_dim 128, two CTAs per SM.  Where the grid and shared memory give an SM more than two, half
// the tiles in 64 registers let four run side by side, so that one's softmax covers the others' loads: eight layers of 32 sequences
// of 191 positions with 32 heads, 1024 CTAs of 42 KB: 1318 -> 1236 us per pass (one tile 1275 us, three CTAs 1282 us).  A grid that
// two CTAs per SM hold at once has no use for more and loses the loads in flight: 64 CTAs, 557 -> 570 us per pass.
template <int HC, int UN>
static int attn_mm_go(const AttnMmP & p, dim3 grid, size_t smem, bool pdl, cudaStream_t st) {
    static bool attr_done[16] = {false};
    int dev = 0;
    PI_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 16 && !attr_done[dev]) {
        PI_CUDA(cudaFuncSetAttribute(k_attention_mm<HC, UN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AM_SMEM_MAX));
        attr_done[dev] = true;
    }
    PI_CUDA(launch_k(k_attention_mm<HC, UN>, grid, dim3(AM_THREADS), smem, st, pdl, p));
    return PI_OK;
}

int launch_attention_mm(const AttnArgs & a, cudaStream_t st) {
    if (!attention_mm_takes(a)) return PI_ERR_UNSUPPORTED;
    AttnMmP p;
    p.q = a.q; p.k = a.k; p.v = a.v; p.k_cache = a.k_cache; p.v_cache = a.v_cache; p.seq = a.seq; p.pos = a.pos; p.T = a.T;
    p.n_head = a.n_head; p.n_head_kv = a.n_head_kv; p.n_ctx = a.n_ctx; p.cs = a.cs; p.neox = a.neox;
    p.q_stride = a.q_stride ? a.q_stride : (int64_t)a.n_head * a.head_dim;
    p.kv_stride = a.kv_stride ? a.kv_stride : (int64_t)a.n_head_kv * a.head_dim;
    p.out = a.out; p.out_act = a.out_act; p.out_act_type = a.out_act_type;
    p.chunk = a.store_mode != 0;
    p.stored = p.chunk && a.T > AM_OWN_STORE;
    size_t smem = attn_mm_smem(a, &p.P, &p.R);
    if (p.stored) PI_CUDA(launch_k(k_kv_store, dim3((unsigned)((a.n_head_kv * a.head_dim / 2 + 255) / 256), a.T), dim3(256), 0, st, a.pdl, p, a.head_dim));
    const dim3 grid = p.chunk ? dim3(a.n_head, (a.T + 15) / 16) : dim3(a.n_head_kv * ((a.n_head / a.n_head_kv + 15) / 16), a.T);
    // CTAs that can have an SM each do: placed early, while the kernel before this one holds other SMs, two would share one (eight sequences of the
    // 70B shape, three layers 536 -> 525 us a step; 32 tokens at position 991, 32 heads of 128, four layers 533 -> 486).
    if ((int64_t)grid.x * grid.y <= sm_count() && smem < AM_SMEM_MAX / 2 + 8192) smem = AM_SMEM_MAX / 2 + 8192;
    if (a.head_dim == 64) return attn_mm_go<2, 4>(p, grid, smem, a.pdl, st);
    return smem <= AM_SMEM_MAX / 3 && (int64_t)grid.x * grid.y > 2 * sm_count() ? attn_mm_go<4, 2>(p, grid, smem, a.pdl, st) : attn_mm_go<4, 4>(p, grid, smem, a.pdl, st);
}

}  // namespace pi
