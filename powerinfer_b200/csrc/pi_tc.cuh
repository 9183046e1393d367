// tcgen05 (fifth-generation tensor cores) primitives and what the kernels that use them share.
//
// Operands lie in shared memory, named by 64-bit descriptors; sums lie in tensor memory (128 lanes x 512 columns of 32 bits per SM).
// One thread issues the products; tcgen05.commit makes an mbarrier complete when all products issued before it are done.
#pragma once
#include <cuda.h>

#include "pi_common.cuh"

namespace pi {

// 2-dimensional tensor map (pi_mm_wide.cu): rows of `cols` elements, `pitch` bytes apart, in boxes of box_cols x box_rows; what lies past the
// ends reads as zeros
int tensor_map(CUtensorMap * m, CUtensorMapDataType type, const void * base, int64_t cols, int64_t rows, int64_t pitch, int box_cols, int box_rows, CUtensorMapSwizzle swizzle);
// the tile of `map` at columns x.., rows y.. (x times the element size a multiple of 16 bytes)
__device__ __forceinline__ void tma_tile(uint32_t dst, const CUtensorMap * map, int x, int y, uint64_t * bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 :: "r"(dst), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar)) : "memory");
}
// the map itself on its way to the SM
__device__ __forceinline__ void tma_map(const CUtensorMap * map) { asm volatile("prefetch.tensormap [%0];" :: "l"(map) : "memory"); }
// ---- tensor memory: allocated by one whole warp, which writes the address to shared memory; given back by the same warp
__device__ __forceinline__ void tc_alloc(uint32_t * slot, unsigned columns) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(slot)), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(uint32_t tmem, unsigned columns) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(columns) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after()  { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// shared memory written by st.shared is read by the tensor cores, which go through another proxy
__device__ __forceinline__ void tc_fence_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Products are issued by one elected lane of a warp that is not divergent (addresses and descriptors stay in uniform registers: a branch
// on the lane number cost 300 clocks per product).  D[128 x N] = A[128 x 16] * B[N x 16] of halves, or with `accumulate` D += A * B.
__device__ __forceinline__ void tc_mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
    asm volatile("{\n .reg .pred e, p;\n elect.sync _|e, 0xffffffff;\n setp.ne.u32 p, %4, 0;\n @e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
                 :: "r"(d), "l"(a), "l"(b), "r"(idesc), "r"((unsigned)accumulate) : "memory");
}
// the same with A in tensor memory: 128 lanes x 8 columns of two halves
__device__ __forceinline__ void tc_mma_f16_ta(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, bool accumulate) {
    asm volatile("{\n .reg .pred e, p;\n elect.sync _|e, 0xffffffff;\n setp.ne.u32 p, %4, 0;\n @e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
                 :: "r"(d), "r"(a), "l"(b), "r"(idesc), "r"((unsigned)accumulate) : "memory");
}
// the barrier completes when all products that this warp's elected lane has issued are done
__device__ __forceinline__ void tc_commit(uint64_t * bar) {
    asm volatile("{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" :: "r"(smem_u32(bar)) : "memory");
}
// instruction descriptor: 128 x n, halves, FP32 sums; b_mn: B lies with its columns, not K, contiguous
__host__ __device__ constexpr uint32_t tc_idesc(int n, bool b_mn) {
    return (1u << 4) | (b_mn ? 1u << 16 : 0u) | ((uint32_t)(n >> 3) << 17) | (8u << 24);
}
// Operands in 128-byte rows whose 16-byte pieces are permuted by the row's number in groups of 8 (piece ^ row: the 128-byte swizzle), from
// 1024-byte boundaries.  K-major: a row is 64 values of K; a step of 16 in K is 32 bytes on.  MN-major: a row is 64 values of M or N at
// one k, 8 k take 1024 bytes, the next 64 values of M or N begin mn_step bytes on; a step of 16 in K is 2048 bytes on.
__device__ __forceinline__ uint64_t tc_desc_k(uint32_t addr) { return (uint64_t)((addr >> 4) & 0x3FFFu) | 1ull << 16 | 64ull << 32 | 1ull << 46 | 2ull << 61; }
__device__ __forceinline__ uint64_t tc_desc_mn(uint32_t addr, uint32_t mn_step) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (uint64_t)(mn_step >> 4) << 16 | 64ull << 32 | 1ull << 46 | 2ull << 61;
}
// 32 lanes (those of this warp's quarter: warp % 4) x 16 columns into registers; returns when they are there.  (Load and wait in ONE statement:
// registers that pass through a wait of their own were copied each time, which cost more than the wait.)
__device__ __forceinline__ void tc_ld16(float (&v)[16], uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\ttcgen05.wait::ld.sync.aligned;"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]) : "r"(addr));
}

__device__ __forceinline__ void tc_ld8(float (&v)[8], uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\ttcgen05.wait::ld.sync.aligned;"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "r"(addr));
}
// 16 columns back; tc_wait_st: this warp's stores are there
__device__ __forceinline__ void tc_st16(uint32_t addr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 :: "r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---- The rows that the masks name, dealt to `groups` in equal contiguous ranges by rank: rank range [lo, hi) of group `grp`, its row
// numbers to rows[0 .. hi - lo).  All THREADS threads call it, s_warp holds THREADS / 32 words; returns the number of active rows.
template <int THREADS>
__device__ __forceinline__ int tc_active_rows(const uint32_t * masks, int nrows, int grp, int groups, int * s_warp, int * rows, int & lo, int & hi) {
    constexpr int KEEP = 4;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_chunks = (nrows + 31) / 32, per = (n_chunks + THREADS - 1) / THREADS;
    const int c0 = min(tid * per, n_chunks), c1 = min(c0 + per, n_chunks);
    auto word = [&](int c) {
        const uint32_t m = __ldcg(masks + c);
        const int left = nrows - c * 32;                              // bits beyond the last row never count
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
    for (int w = 0; w < THREADS / 32; w++) { if (w < warp) before += s_warp[w]; total += s_warp[w]; }
    total = __shfl_sync(0xffffffffu, total, 0);
    lo = (int)((unsigned)total * (unsigned)grp / (unsigned)groups);   // (up to 262144 rows, 148 groups: 32 bits)
    hi = (int)((unsigned)total * (unsigned)(grp + 1) / (unsigned)groups);
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
    return total;
}

}  // namespace pi
