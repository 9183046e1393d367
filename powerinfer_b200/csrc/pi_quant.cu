// Block formats of the hot path: Q4_0 weights (quantise, re-layout, dequantise) and the Q8_0 / FP16
// forms activations take before a mat-vec.  All kernels are HBM- or latency-bound byte shuffles.
#include "pi_common.cuh"

namespace pi {

static constexpr int QK = 32;

// ------------------------------------------------------------------------------------------------
// quantize_row_q4_0_reference (ggml-quants.c:428-463).  One warp per block of 32 values, lane = value.
// The reference keeps the FIRST value of largest magnitude; ties are resolved to the lowest lane.
__global__ void k_quantize_q4_0(const float * __restrict__ x, uint8_t * __restrict__ q, int64_t nblocks) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t b = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); b < nblocks; b += warps) {
        const float v = x[b * QK + lane];
        float amax = fabsf(v);
        int   arg  = lane;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float oa = __shfl_xor_sync(0xffffffffu, amax, o);
            const int   ol = __shfl_xor_sync(0xffffffffu, arg, o);
            if (oa > amax || (oa == amax && ol < arg)) { amax = oa; arg = ol; }
        }
        const float mx = __shfl_sync(0xffffffffu, v, arg);
        const float d  = mx / -8.0f;
        const float id = d != 0.0f ? 1.0f / d : 0.0f;
        // two roundings as in the reference (x*id, then +8.5): keep the compiler from fusing them into one FMA
        int qi = (int)(int8_t)__fadd_rn(__fmul_rn(v, id), 8.5f);   // float -> int8 truncates toward zero
        qi = qi > 15 ? 15 : qi;
        const int hi = __shfl_down_sync(0xffffffffu, qi, 16);
        uint8_t * blk = q + b * 18;
        if (lane == 0) *reinterpret_cast<__half *>(blk) = __float2half_rn(d);
        if (lane < 16) blk[2 + lane] = (uint8_t)((qi & 0xF) | (hi << 4));
    }
}

int launch_quantize_q4_0(const float * x, void * q4, int64_t nrows, int64_t ncols, cudaStream_t st) {
    const int64_t nblocks = nrows * (ncols / QK);
    if (nblocks == 0) return PI_OK;
    const int grid = (int)imin64((nblocks + 7) / 8, (int64_t)sm_count() * 16);
    k_quantize_q4_0<<<grid, 256, 0, st>>>(x, (uint8_t *)q4, nblocks);
    PI_LAUNCH_CHECK("k_quantize_q4_0");
    return PI_OK;
}

// ------------------------------------------------------------------------------------------------
// ggml layout: row = nb x {fp16 d; uint8 qs[16]}.  Planar layout: row = nb x qs[16] then nb x fp16 d.
// One thread per block; 2-byte accesses on the ggml side (blocks are only 2-byte aligned).
__global__ void k_q4_0_repack(const uint8_t * __restrict__ src, uint8_t * __restrict__ dst, int64_t nrows, int nb) {
    const int64_t total = nrows * nb;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = i / nb;
        const int b = (int)(i - r * nb);
        const uint16_t * s = reinterpret_cast<const uint16_t *>(src + (r * nb + b) * 18);
        uint8_t * row = dst + r * (int64_t)nb * 18;
        uint16_t w[9];
#pragma unroll
        for (int j = 0; j < 9; j++) w[j] = s[j];
        uint4 qv;
        qv.x = w[1] | ((uint32_t)w[2] << 16);
        qv.y = w[3] | ((uint32_t)w[4] << 16);
        qv.z = w[5] | ((uint32_t)w[6] << 16);
        qv.w = w[7] | ((uint32_t)w[8] << 16);
        reinterpret_cast<uint4 *>(row)[b] = qv;
        reinterpret_cast<uint16_t *>(row + (int64_t)nb * 16)[b] = w[0];
    }
}

int launch_q4_0_repack(const void * src, void * dst, int64_t nrows, int64_t ncols, cudaStream_t st) {
    const int nb = (int)(ncols / QK);
    const int64_t total = nrows * nb;
    if (total == 0) return PI_OK;
    const int grid = (int)imin64((total + 255) / 256, (int64_t)sm_count() * 16);
    k_q4_0_repack<<<grid, 256, 0, st>>>((const uint8_t *)src, (uint8_t *)dst, nrows, nb);
    PI_LAUNCH_CHECK("k_q4_0_repack");
    return PI_OK;
}

// dequantize_row_q4_0 (ggml-quants.c:1074-1092) from the planar layout; one thread per block
__global__ void k_dequantize_q4_0(const uint8_t * __restrict__ q, float * __restrict__ y, int64_t nrows, int nb) {
    const int64_t total = nrows * nb;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = i / nb;
        const int b = (int)(i - r * nb);
        const uint8_t * row = q + r * (int64_t)nb * 18;
        const uint4 qv = reinterpret_cast<const uint4 *>(row)[b];
        const float d = __half2float(reinterpret_cast<const __half *>(row + (int64_t)nb * 16)[b]);
        const uint32_t w[4] = {qv.x, qv.y, qv.z, qv.w};
        float * o = y + (r * nb + b) * QK;
#pragma unroll
        for (int j = 0; j < 16; j++) {
            const uint32_t byte = (w[j >> 2] >> ((j & 3) * 8)) & 0xFFu;
            o[j]      = (float)((int)(byte & 0xF) - 8) * d;
            o[j + 16] = (float)((int)(byte >> 4) - 8) * d;
        }
    }
}

int launch_dequantize_q4_0(const void * q4p, float * y, int64_t nrows, int64_t ncols, cudaStream_t st) {
    const int nb = (int)(ncols / QK);
    const int64_t total = nrows * nb;
    if (total == 0) return PI_OK;
    const int grid = (int)imin64((total + 255) / 256, (int64_t)sm_count() * 16);
    k_dequantize_q4_0<<<grid, 256, 0, st>>>((const uint8_t *)q4p, y, nrows, nb);
    PI_LAUNCH_CHECK("k_dequantize_q4_0");
    return PI_OK;
}

// ------------------------------------------------------------------------------------------------
// quantize_row_q8_0, the AVX2 branch the CPU path runs (ggml-quants.c:702-760):
//   d = amax / 127, id = amax != 0 ? 127 / amax : 0, q = round-to-nearest-even(x * id), d stored as FP16.
// One warp per block, lane = value.
__device__ __forceinline__ void q8_block(float v, int & q, float & d16, int & sum) {
    const float amax = warp_max(fabsf(v));
    const float d  = amax / 127.0f;
    const float id = amax != 0.0f ? 127.0f / amax : 0.0f;
    q = __float2int_rn(v * id);
    d16 = __half2float(__float2half_rn(d));
    sum = warp_sum_i(q);
}

__global__ void k_quantize_q8_0_ggml(const float * __restrict__ x, uint8_t * __restrict__ q8, int64_t nblocks) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t b = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); b < nblocks; b += warps) {
        int q, s; float d16;
        q8_block(x[b * QK + lane], q, d16, s);
        uint8_t * blk = q8 + b * 34;
        if (lane == 0) *reinterpret_cast<__half *>(blk) = __float2half_rn(d16);
        reinterpret_cast<int8_t *>(blk + 2)[lane] = (int8_t)q;
    }
}

int launch_quantize_q8_0_ggml(const float * x, void * q8, int64_t nrows, int64_t ncols, cudaStream_t st) {
    const int64_t nblocks = nrows * (ncols / QK);
    if (nblocks == 0) return PI_OK;
    const int grid = (int)imin64((nblocks + 7) / 8, (int64_t)sm_count() * 16);
    k_quantize_q8_0_ggml<<<grid, 256, 0, st>>>(x, (uint8_t *)q8, nblocks);
    PI_LAUNCH_CHECK("k_quantize_q8_0_ggml");
    return PI_OK;
}

// ------------------------------------------------------------------------------------------------
// Activation planes (see Act in pi_common.cuh)
size_t act_bytes(int wtype, int64_t n, int T) {
    auto up = [](size_t v) { return (v + 255) & ~size_t(255); };
    if (wtype == PI_TYPE_Q4_0) {
        const size_t nb = (size_t)(n / QK);
        return 2 * up((size_t)T * nb * 16) + 2 * up((size_t)T * nb * 4);
    }
    return up((size_t)T * n * 2);
}

ActBuf act_carve(int wtype, int64_t n, int T, char ** p) {
    auto take = [&](size_t bytes) { char * r = *p; *p += (bytes + 255) & ~size_t(255); return r; };
    ActBuf a;
    if (wtype == PI_TYPE_Q4_0) {
        const size_t nb = (size_t)(n / QK);
        a.lo = (uint4 *)take((size_t)T * nb * 16);
        a.hi = (uint4 *)take((size_t)T * nb * 16);
        a.d  = (float *)take((size_t)T * nb * 4);
        a.s  = (int *)take((size_t)T * nb * 4);
    } else {
        a.h16 = (__half *)take((size_t)T * n * 2);
    }
    return a;
}

// What an operator needs before its weight-streaming kernel, in one launch: activation planes of x, activity bit masks of the predictor
// logits, zeros where nobody else will write, cleared control words.  Each is a few hundred KB at most, so they cost their launches
// (2 us each, two memsets among them); the blocks of the grid are handed to the parts in turn.
struct PrepP {
    const float * x; int n, nb, T; ActBuf act;
    const float * idx; int64_t idx_stride; float threshold; int n_local; const int32_t * bucket; uint32_t * masks;
    float * zero; int64_t n_zero; unsigned int * words; int n_words;
    int g_act, g_mask;                                                // blocks of the first two parts, the others zero
};

template <bool Q4>
__global__ void __launch_bounds__(256) k_prep(const PrepP p) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int b = blockIdx.x;
    pdl_wait();
    pdl_launch();                                                     // (after the wait: a kernel that runs ahead may read weights that came before)
    if (b == 0 && tid < p.n_words) p.words[tid] = 0u;
    if (b < p.g_act) {
        if (Q4) {
            const int64_t n = (int64_t)p.T * p.nb;
            for (int64_t i = (int64_t)b * 8 + warp; i < n; i += (int64_t)p.g_act * 8) {
                int q, s; float d16;
                q8_block(p.x[i * QK + lane], q, d16, s);
                int8_t * plane = reinterpret_cast<int8_t *>(lane < 16 ? p.act.lo + i : p.act.hi + i);
                plane[lane & 15] = (int8_t)q;
                if (lane == 0) { p.act.d[i] = d16; p.act.s[i] = s; }
            }
        } else {
            const int64_t n = (int64_t)p.T * p.n, step = (int64_t)p.g_act * 256;
            int64_t i = (int64_t)b * 256 + tid;
            for (; i + 3 * step < n; i += 4 * step) {
                float v[4];
#pragma unroll
                for (int u = 0; u < 4; u++) v[u] = p.x[i + u * step];
#pragma unroll
                for (int u = 0; u < 4; u++) p.act.h16[i + u * step] = __float2half_rn(v[u]);
            }
            for (; i < n; i += step) p.act.h16[i] = __float2half_rn(p.x[i]);
        }
        return;
    }
    b -= p.g_act;
    if (b < p.g_mask) {                                               // one warp per 32 rows, as in k_compact
        const int n_chunks = (p.n_local + 31) / 32;
        constexpr int UN = 8;                                         // logits in flight per lane
        for (int c = b * 8 + warp; c < n_chunks; c += p.g_mask * 8) {
            const int r = c * 32 + lane;
            bool any = false;
            if (r < p.n_local) {
                const float * row = p.idx + (p.bucket ? p.bucket[r] : r);
                for (int t0 = 0; t0 < p.T; t0 += UN) {
                    float l[UN];
#pragma unroll
                    for (int u = 0; u < UN; u++) l[u] = t0 + u < p.T ? row[(size_t)(t0 + u) * p.idx_stride] : 0.f;
#pragma unroll
                    for (int u = 0; u < UN; u++) any |= t0 + u < p.T && !(l[u] < p.threshold);      // (a NaN logit counts as active)
                }
            }
            const uint32_t m = __ballot_sync(0xffffffffu, any);
            if (lane == 0) p.masks[c] = m;
        }
        return;
    }
    b -= p.g_mask;
    const int64_t step = (int64_t)(gridDim.x - p.g_act - p.g_mask) * 256;
    for (int64_t i = (int64_t)b * 256 + tid; i < p.n_zero; i += step) p.zero[i] = 0.f;
}

int launch_prep(const PrepArgs & a, cudaStream_t st) {
    PrepP p;
    p.x = a.x; p.n = (int)a.n; p.nb = (int)(a.n / QK); p.T = a.T; p.act = a.act;
    p.idx = a.idx; p.idx_stride = a.idx_stride; p.threshold = a.threshold; p.n_local = (int)a.n_local; p.bucket = a.bucket; p.masks = a.masks;
    p.zero = a.zero; p.n_zero = a.zero ? a.n_zero : 0; p.words = a.words; p.n_words = a.words ? a.n_words : 0;
    const bool q4 = a.wtype == PI_TYPE_Q4_0;
    const int64_t most = (int64_t)sm_count() * 8;
    p.g_act = !a.x ? 0 : (int)imin64(q4 ? ((int64_t)a.T * p.nb + 7) / 8 : ((int64_t)a.T * a.n + 1023) / 1024, most);
    p.g_mask = !a.idx ? 0 : (int)imin64((a.n_local + 255) / 256, most);
    const int g_zero = (int)imin64((p.n_zero + 1023) / 1024, most);
    const int grid = p.g_act + p.g_mask + g_zero > 0 ? p.g_act + p.g_mask + g_zero : 1;
    if (q4) PI_CUDA(launch_k(k_prep<true>, dim3(grid), dim3(256), 0, st, true, p));
    else    PI_CUDA(launch_k(k_prep<false>, dim3(grid), dim3(256), 0, st, true, p));
    return PI_OK;
}

// ------------------------------------------------------------------------------------------------
// Coefficients of the Q4_0 axpy (ggml.c:14575-14581): the FFN hidden vector quantised to Q8_0 over blocks of
// 32 consecutive NEURONS; neuron r contributes int8 b = cq[r] with scale cd[r/32].
__global__ void k_neuron_q8(const float * __restrict__ h, int nb, int8_t * __restrict__ cq, float * __restrict__ cd) {
    const int lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x >> 5);
    for (int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); b < nb; b += warps) {
        int q, s; float d16;
        q8_block(h[(int64_t)b * QK + lane], q, d16, s);
        cq[(int64_t)b * QK + lane] = (int8_t)q;
        if (lane == 0) cd[b] = d16;
    }
}

int launch_neuron_q8(const float * h, int64_t n, int8_t * cq, float * cd, cudaStream_t st) {
    const int nb = (int)(n / QK);
    if (nb == 0) return PI_OK;
    const int grid = (int)imin64(((int64_t)nb + 7) / 8, (int64_t)sm_count() * 8);
    k_neuron_q8<<<grid, 256, 0, st>>>(h, nb, cq, cd);
    PI_LAUNCH_CHECK("k_neuron_q8");
    return PI_OK;
}

}  // namespace pi
