// Device helpers shared by the dense nodes: activation planes for the next mat-vec, RoPE.
#pragma once
#include "pi_common.cuh"

namespace pi {

static constexpr int QK = 32;

// (put_act of the one-launch step does the same into shared memory.)
// Emit 8 consecutive values (chunk index c8 = first column / 8) of token t as activation planes.
// Must be called by every lane of a warp (it shuffles); `valid` gates the stores.  With n % 32 == 0 the 4 lanes that
// share a Q8 block are valid or invalid together.
__device__ __forceinline__ void emit_act8(int type, const ActBuf & a, int t, int64_t n, int c8, const float (&v)[8], bool valid) {
    if (type == PI_TYPE_F16) {
        if (!valid) return;
        __half2 h[4];
#pragma unroll
        for (int j = 0; j < 4; j++) h[j] = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
        *reinterpret_cast<uint4 *>(a.h16 + (size_t)t * n + (size_t)c8 * 8) = *reinterpret_cast<uint4 *>(h);
    } else if (type == PI_TYPE_Q4_0) {
        // 4 consecutive threads (lanes 4k..4k+3) hold one block of 32 values
        float amax = 0.f;
#pragma unroll
        for (int j = 0; j < 8; j++) amax = fmaxf(amax, fabsf(v[j]));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        const float d  = amax / 127.0f;
        const float id = amax != 0.0f ? 127.0f / amax : 0.0f;
        int q[8], s = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) { q[j] = __float2int_rn(v[j] * id); s += q[j]; }
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        const int nb = (int)(n / QK);
        const size_t blk = (size_t)t * nb + (c8 >> 2);
        const int part = c8 & 3;                                  // which 8 of the 32
        uint2 packed;
        packed.x = (uint32_t)(q[0] & 0xFF) | ((uint32_t)(q[1] & 0xFF) << 8) | ((uint32_t)(q[2] & 0xFF) << 16) | ((uint32_t)(q[3] & 0xFF) << 24);
        packed.y = (uint32_t)(q[4] & 0xFF) | ((uint32_t)(q[5] & 0xFF) << 8) | ((uint32_t)(q[6] & 0xFF) << 16) | ((uint32_t)(q[7] & 0xFF) << 24);
        if (!valid) return;
        uint2 * plane = reinterpret_cast<uint2 *>(part < 2 ? a.lo + blk : a.hi + blk);
        plane[part & 1] = packed;
        if (part == 0) { a.d[blk] = __half2float(__float2half_rn(d)); a.s[blk] = s; }
    }
}

// one pair of ggml_rope_custom: products and sums are rounded separately, as the CPU build does
__device__ __forceinline__ void rope_pair(float x0, float x1, float c, float s, float & o0, float & o1) {
    o0 = __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s));
    o1 = __fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c));
}

}  // namespace pi
