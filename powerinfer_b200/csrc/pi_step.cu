// One decode step of ONE sequence as ONE launch: all layers and the lm head in a persistent, cooperatively launched grid of one
// CTA per SM (what llama_decode -> llm_build_{llama,falcon,opt} -> ggml_graph_compute runs node by node: llama.cpp:6764-7006).
//
// What bounds a step is the chain: every node needs the whole vector the node before it made, a layer's bytes are spread over
// 8 dependent nodes of 5-60 MB, and a kernel per node drains and refills the memory pipeline at every boundary (a layer of the
// 70B shape: 73 us for 207 MB, 32 us at the copy rate).  Here
//   weights   copying warps stream the rows of THIS SM (QKV, out-proj, fc1, fc2, gathered rows of every layer, lm head) through one
//             shared-memory ring, in the order the step needs them and without regard to where the arithmetic is: weights depend
//             on nothing, so the ring fills while the computing warps wait for another CTA's values.  At most `window` slots are
//             on their way at a time: the queue in front of the memory stays short, and with it the latency of the small reads
//             below (28 MB requested at once by all SMs delay a small read by 4 us);
//   values    travel between CTAs as words that carry their own validity: {float, number of the layer} in 8 bytes, {16 bits, 16
//             bits of the number} or {8 mask bits, 24 bits} in 4.  A consumer polls the words it needs; there is no barrier
//             across the grid, no fence and no flag, one trip through L2 per hand-over.  Norms are computed by every CTA for
//             itself (the sum of squares costs less than a hand-over);
//   sparse    the gather takes rows by rank from the predictor's masks, evenly over the CTAs; the axpy takes (1024-column slice,
//             group of whole 32-neuron blocks); partial vectors are added in group order by the CTA that owns the columns.  No
//             atomics on values, every sum in a fixed order: same bits every run.
// A word is overwritten two layers later at the earliest (buffers alternate by the parity of the layer).  By then every CTA has
// read it: each CTA owns at least one row of the out-projection, whose whole output every later layer's words depend on, and it
// computes that row behind all its reads of the layer before.
// Every wait ends (pi_engine_set_wait_cycles): where a copying warp has waited for about a second since the last CTA of the step was seen to
// run, or 64 times as long before that (a kernel of another stream may hold an SM), it ends the waits of all, and the step finishes with
// wrong values, the greedy id -1 and bit 3 of the status word (12 ms for 8 layers of the 70B shape).  From then on the computing warps go on
// without the copying warps' leave.  So what an address is made from holds whoever is late: the gather's rows have a place of their own, in
// which nothing but row numbers stands, and the copying warps get the number of rows and that of slots in one word.
//
// The arithmetic of four nodes stands here a second time, with other inputs and outputs: attention_head (k_attention_row), norm_phase
// (k_norm), put_act (emit_act8), axpy_phase (k_ffn_rows, k_axpy_rows).  A change of one is a change of both; steps by this kernel and by
// the launch sequence are compared in the tests.
#include "pi_rows.cuh"
#include "pi_step.cuh"

#include <cuda.h>

#include <algorithm>
#include <cstdlib>

namespace pi {

typedef unsigned long long u64;

// ------------------------------------------------------------------------------------------------ words that carry their own validity
__device__ __forceinline__ void ld2(const u64 * p, u64 & a, u64 & b) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ u64 ld1(const u64 * p) {
    u64 a;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
    return a;
}
__device__ __forceinline__ uint4 ld4(const uint32_t * p) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ldw(const uint32_t * p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st1(u64 * p, float v, unsigned tag) {
    const u64 w = (u64)tag << 32 | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" :: "l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ void stw(uint32_t * p, uint32_t v) { asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" :: "l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ void mbar_arrive_n(uint64_t * bar, unsigned n) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" :: "r"(smem_u32(bar)), "r"(n) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t * bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool fresh(u64 w, unsigned tag) { return (unsigned)(w >> 32) == tag; }
__device__ __forceinline__ float val(u64 w) { return __uint_as_float((unsigned)w); }
__device__ __forceinline__ void bar_ct() { asm volatile("bar.sync 1, 512;" ::: "memory"); }

// ------------------------------------------------------------------------------------------------ what every phase reads, in shared memory
// (Shared memory takes nearly all of an SM's storage: what is spilled to local memory comes back from L2.  The phases are functions of
// their own that take two or three values and find the rest here, so that none of them keeps another's values alive.)
extern __shared__ __align__(128) unsigned char smem[];                // ring | scratch, see step_plan
static __shared__ StepP s_p;
static __shared__ StepLayer s_layer[2];                               // this layer's and the next one's
static __shared__ int s_first[ST_N_MAT], s_rows[ST_N_MAT], s_slots[ST_N_MAT];   // this CTA's rows of every matrix, and the ring slots they take
static __shared__ __align__(8) uint64_t s_full[ST_MAX_SLOTS], s_empty[ST_MAX_SLOTS], s_listed, s_taken, s_done;   // s_done: the computing warps have waited for the last time; s_listed: the gather's rows of this layer are listed; s_taken: the copying warps have read them
static __shared__ double s_dred[ST_WARPS];
static __shared__ int s_warp[ST_WARPS];
static __shared__ int s_kb, s_ke, s_kz, s_col0, s_ncol;                 // s_col0, s_ncol: the columns of the residual stream that this CTA adds up
static __shared__ volatile int s_dead;                                // 1: a wait ran out, nobody waits any more; 2: all waits of this CTA ended well
static __shared__ unsigned int s_step;
static __shared__ volatile unsigned int s_gather;                     // rows and slots (in the upper half) of the gather, for the copying warps

__device__ __forceinline__ int mat_slots(const StepMat & m, int nrow) { return m.pieces > 1 ? nrow * m.pieces : (nrow + m.rps - 1) / m.rps; }
__device__ __forceinline__ uint32_t * sh_mask() { return reinterpret_cast<uint32_t *>(smem + s_p.off_b); }
__device__ __forceinline__ int * sh_pref() { return reinterpret_cast<int *>(smem + s_p.off_b) + s_p.F / 32; }
__device__ __forceinline__ int * sh_list() { return sh_pref() + s_p.F / 32 + 1; }                    // [4][ST_LIST]
__device__ __forceinline__ int * sh_rows() { return reinterpret_cast<int *>(smem + s_p.off_rows); }      // this CTA's rows of the gather
__device__ __forceinline__ float * sh_part() { return reinterpret_cast<float *>(smem + s_p.off_part); }

// Waits.  The kernel's code is walked through once per layer and has to stay in the instruction cache (at 170 KB a layer, every phase ran at
// a third of its speed): what is not there at the first look goes to a function.
// Only the copying warps' waits have a clock: where the step does not go on, the ring stays full and they wait.  The computing warps look
// whether the step has been ended, by their CTA or another: a clock and a count of the running CTAs in the dozen places where they wait cost
// up to 4 % of a step (registers spill, polls get longer).
// (The look at the word in L2 costs nothing: 80 layers of the 70B shape 180.8 tok/s with it, 178.8 where only s_dead is read.)
__device__ __forceinline__ bool wait_over(int & polls) {
    if ((++polls & 63) != 0) return false;
    if (s_dead) return true;
    if (ldw(s_p.abort) != s_step + 1u) return false;
    s_dead = 1;
    return true;
}
__device__ __noinline__ bool wait_bar_slow(uint64_t * bar, unsigned parity) {
    int tries = 0;
    while (!mbar_try_wait(bar, parity)) if ((++tries & 7) == 0 && s_dead) return false;
    return true;
}
__device__ __forceinline__ bool wait_bar(uint64_t * bar, unsigned parity) { return mbar_test(bar, parity) || wait_bar_slow(bar, parity); }
__device__ __forceinline__ void end_step() { stw(s_p.abort, s_step + 1u); atomicOr(s_p.status, 8u); }
__device__ __noinline__ bool timed_bar_slow(uint64_t * bar, unsigned parity) {
    long long from = clock64();
    bool placed = false;                                              // all CTAs of the step run
    for (int i = 1; !mbar_try_wait(bar, parity); i++) {
        if (s_dead) return false;
        if ((i & s_p.look) != 0) continue;
        const long long now = clock64();
        if (!placed && ldw(s_p.arrived) == (s_step + 1u) * gridDim.x) { placed = true; from = now; }
        if (now - from <= (placed ? s_p.limit : 64 * s_p.limit) && ldw(s_p.abort) != s_step + 1u) continue;
        if (atomicCAS(const_cast<int *>(&s_dead), 0, 1) == 0) end_step();
        return false;
    }
    return true;
}
__device__ __forceinline__ bool timed_bar(uint64_t * bar, unsigned parity) { return mbar_test(bar, parity) || timed_bar_slow(bar, parity); }
// until each of the n words carries the number; returns the last one
__device__ __noinline__ u64 wait_words(const u64 * p, int n, unsigned tag) {
    u64 x = 0ull;
    for (int i = 0; i < n; i++) {
        int polls = 0;
        for (x = ld1(p + i); !fresh(x, tag); x = ld1(p + i)) if (wait_over(polls)) break;
    }
    return x;
}
// the same for four 4-byte words whose number stands above the lowest `bits` bits
__device__ __noinline__ uint4 wait_words4(const uint32_t * p, int bits, unsigned tag) {
    int polls = 0;
    uint4 v = ld4(p);
    while (((v.x ^ tag) | (v.y ^ tag) | (v.z ^ tag) | (v.w ^ tag)) >> bits) { if (wait_over(polls)) break; v = ld4(p); }
    return v;
}
__device__ __forceinline__ float wait_val(const u64 * s, unsigned tag) {
    u64 x = ld1(s);
    if (!fresh(x, tag)) x = wait_words(s, 1, tag);
    return val(x);
}

// ------------------------------------------------------------------------------------------------ rows from the ring

// two of the FP32 sums of products of FP16 pairs; the hardware takes the halves as they are (a conversion to FP32 first costs a third more)
__device__ __forceinline__ void fma_h2(float & a, float & b, uint32_t w, uint32_t x) {
    asm("{\n .reg .b16 w0, w1, x0, x1;\n mov.b32 {w0, w1}, %2;\n mov.b32 {x0, x1}, %3;\n fma.rn.f32.f16 %0, w0, x0, %0;\n fma.rn.f32.f16 %1, w1, x1, %1;\n}"
        : "+f"(a), "+f"(b) : "r"(w), "r"(x));
}

// What one lane holds of the activation while rows go by: `upt` units of a row (F16: 8 columns, Q4_0: a block of 32).  dot: N rows, whose
// reads travel together.  nq: units of the piece of a row that lies in the slot.
template <int WT, int UPT> struct XReg;
template <int UPT> struct XReg<PI_TYPE_F16, UPT> {
    uint4 x[UPT];
    __device__ __forceinline__ void load(const unsigned char * xs, int, int u0, int step, bool last_ok) {
#pragma unroll
        for (int j = 0; j < UPT; j++) x[j] = j < UPT - 1 || last_ok ? reinterpret_cast<const uint4 *>(xs)[u0 + j * step] : make_uint4(0u, 0u, 0u, 0u);
    }
    template <int N>
    __device__ __forceinline__ void dot(const unsigned char * row, int n, int stride, int, int u0, int step, bool last_ok, float (&v)[N]) const {
        float a[N], b[N];
#pragma unroll
        for (int r = 0; r < N; r++) { a[r] = 0.f; b[r] = 0.f; }
#pragma unroll
        for (int j = 0; j < UPT; j++) {
            if (j == UPT - 1 && !last_ok) break;
            uint4 w[N];
#pragma unroll
            for (int r = 0; r < N; r++) w[r] = reinterpret_cast<const uint4 *>(row + (r < n ? r * stride : 0))[u0 + j * step];
#pragma unroll
            for (int r = 0; r < N; r++) { fma_h2(a[r], b[r], w[r].x, x[j].x); fma_h2(a[r], b[r], w[r].y, x[j].y); fma_h2(a[r], b[r], w[r].z, x[j].z); fma_h2(a[r], b[r], w[r].w, x[j].w); }
        }
#pragma unroll
        for (int r = 0; r < N; r++) v[r] = a[r] + b[r];
    }
};
template <int UPT> struct XReg<PI_TYPE_Q4_0, UPT> {
    uint4 lo[UPT], hi[UPT]; float d[UPT]; int s8[UPT];                 // int8 of the block's two halves, scale, sum
    __device__ __forceinline__ void load(const unsigned char * xs, int units, int u0, int step, bool last_ok) {
#pragma unroll
        for (int j = 0; j < UPT; j++) {
            lo[j] = hi[j] = make_uint4(0u, 0u, 0u, 0u); d[j] = 0.f; s8[j] = 0;
            if (j < UPT - 1 || last_ok) {
                const int u = u0 + j * step;
                lo[j] = reinterpret_cast<const uint4 *>(xs)[u];
                hi[j] = reinterpret_cast<const uint4 *>(xs)[units + u];
                const uint2 m = reinterpret_cast<const uint2 *>(xs + units * 32)[u];
                d[j] = __uint_as_float(m.x); s8[j] = (int)m.y;
            }
        }
    }
    template <int N>
    __device__ __forceinline__ void dot(const unsigned char * row, int n, int stride, int nq, int u0, int step, bool last_ok, float (&v)[N]) const {
#pragma unroll
        for (int r = 0; r < N; r++) v[r] = 0.f;
#pragma unroll
        for (int j = 0; j < UPT; j++) {
            if (j == UPT - 1 && !last_ok) break;
            const int u = u0 + j * step;
            uint4 q[N]; __half d4[N];
#pragma unroll
            for (int r = 0; r < N; r++) {
                q[r] = reinterpret_cast<const uint4 *>(row + (r < n ? r * stride : 0))[u];
                d4[r] = reinterpret_cast<const __half *>(row + (r < n ? r * stride : 0) + nq * 16)[u];
            }
#pragma unroll
            for (int r = 0; r < N; r++) v[r] = fmaf((float)q4_block_dot(q[r], lo[j], hi[j], s8[j]), __half2float(d4[r]) * d[j], v[r]);
        }
    }
};

// the warp's sums of n of N values to s[0], s[step], ...: they are halved over the lanes as they are added (four: 6 shuffles, not 20)
template <int N>
__device__ __forceinline__ void store_sums(const float (&v)[N], float * s, int step, int n, int lane) {
    const bool h1 = lane & 16, h0 = lane & 8;
    float c;
    int r;
    if (N == 4) {
        float a = h1 ? v[N / 2] : v[0], b = h1 ? v[N - 1] : v[N / 4];
        a += __shfl_xor_sync(0xffffffffu, h1 ? v[0] : v[N / 2], 16);
        b += __shfl_xor_sync(0xffffffffu, h1 ? v[N / 4] : v[N - 1], 16);
        c = (h0 ? b : a) + __shfl_xor_sync(0xffffffffu, h0 ? a : b, 8);
        r = (h1 ? 2 : 0) + (h0 ? 1 : 0);
    } else if (N == 1) {
        c = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16);
        c += __shfl_xor_sync(0xffffffffu, c, 8);
        r = 0;
    } else {
        c = (h1 ? v[N - 1] : v[0]) + __shfl_xor_sync(0xffffffffu, h1 ? v[0] : v[N - 1], 16);
        c += __shfl_xor_sync(0xffffffffu, c, 8);
        r = h1 ? 1 : 0;
    }
    c += __shfl_xor_sync(0xffffffffu, c, 4);
    c += __shfl_xor_sync(0xffffffffu, c, 2);
    c += __shfl_xor_sync(0xffffffffu, c, 1);
    if ((lane & (32 / N - 1)) == 0 && r < n) s[r * step] = c;
}

// Rows of matrix `mi` in slots k0 .. of the ring.  A slot (up to four whole rows, or one piece of a row) is the work of a team of `wpr`
// warps (slot i of the call goes to team i % teams), each lane with the same columns of every row: its part of the activation stays in
// registers, shared memory is read once per weight, and a warp has one wait, one hand-back and one sum over its lanes per slot; the next
// slot is looked at before that sum, whose latency covers the look.  The sums of row r go to sh_part[r * parts ..].  Ends with a barrier
// of the computing warps.
template <int WT, int UPT, int N>                                      // N rows at a time: a slot holds at most as many (mat_plan)
__device__ __noinline__ void consume_t(int mi, unsigned k0, int nrow, const unsigned char * xs) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const StepMat & m = s_p.mat[mi];
    const int units = m.units, R = m.rps, P = m.pieces, wpr = m.wpr, teams = ST_WARPS >> __popc(wpr - 1), stride = (int)m.row_bytes, slot = s_p.slot_bytes, parts = P * wpr;
    const unsigned ring = (unsigned)s_p.n_slots;
    const int team = warp >> __popc(wpr - 1), part = warp & (wpr - 1), pc = team & (P - 1), first = pc * m.punits, nq = min(m.punits, units - first);
    const int u0 = part * 32 + lane, step = wpr * 32;
    const bool last_ok = u0 + (UPT - 1) * step < nq;
    XReg<WT, UPT> x;
    x.load(xs, units, first + u0, step, last_ok);
    const int pshift = __popc(P - 1);
    float * s_part = sh_part() + pc * wpr + part;
    const int nslots = P > 1 ? nrow * P : (nrow + R - 1) / R;   // (a wait ran out: nothing comes any more)
    const unsigned k = k0 + team, round = k / ring;
    unsigned s = k - round * ring, par = round & 1u;
    if (team < nslots) wait_bar(s_full + s, par);
#pragma unroll 1
    for (int i = team; i < nslots; i += teams) {
        const int row0 = P > 1 ? i >> pshift : i * R, n = N == 1 ? 1 : min(R, nrow - row0);
        float v[N];
        x.template dot<N>(smem + s * slot, n, stride, nq, u0, step, last_ok, v);
        __syncwarp();
        if (lane == 0) mbar_arrive_n(s_empty + s, (unsigned)teams);
        s += teams;
        if (s >= ring) { s -= ring; par ^= 1u; }
        const bool ready = i + teams >= nslots || mbar_test(s_full + s, par);
        store_sums<N>(v, s_part + row0 * parts, parts, n, lane);
        if (!ready) wait_bar_slow(s_full + s, par);
    }
    bar_ct();
}

template <int WT>
__device__ __noinline__ void consume(int mi, unsigned k0, int nrow, const unsigned char * xs) {
    switch (s_p.mat[mi].upt) {
        case 1:  consume_t<WT, 1, 4>(mi, k0, nrow, xs); break;
        case 2:  consume_t<WT, 2, 4>(mi, k0, nrow, xs); break;
        case 3:  if (s_p.mat[mi].rps == 1) consume_t<WT, 3, 1>(mi, k0, nrow, xs); else consume_t<WT, 3, 2>(mi, k0, nrow, xs); break;
        default: if (s_p.mat[mi].rps == 1) consume_t<WT, 4, 1>(mi, k0, nrow, xs); else consume_t<WT, 4, 2>(mi, k0, nrow, xs); break;
    }
}

__device__ __forceinline__ float row_total(int mi, int r) {
    const int parts = s_p.mat[mi].wpr * s_p.mat[mi].pieces;
    const float * s = sh_part() + r * parts;
    float v = s[0];
#pragma unroll 4
    for (int q = 1; q < parts; q++) v += s[q];
    return v;
}

// all rows of this CTA: as many at a time as have room for their sums (`chunk`: whole slots).  done(row, sum) for every row.
__device__ __forceinline__ unsigned slot_of(int mi, int row) { return (unsigned)(s_p.mat[mi].pieces > 1 ? row * s_p.mat[mi].pieces : row / s_p.mat[mi].rps); }
template <int WT, typename F>
__device__ __forceinline__ void rows_of(int mi, unsigned kbase, const unsigned char * xs, F done) {
    const int n = s_rows[mi], chunk = s_p.mat[mi].chunk;
#pragma unroll 1
    for (int c0 = 0; c0 < n; c0 += chunk) {
        const int nc = min(chunk, n - c0);
        consume<WT>(mi, kbase + slot_of(mi, c0), nc, xs);
#pragma unroll 1
        for (int t = threadIdx.x; t < nc; t += ST_CT) done(c0 + t, row_total(mi, t));
        bar_ct();
    }
}

// ------------------------------------------------------------------------------------------------ vectors

// 8 normalised (or raw) values, columns c8 * 8 .., as the next product's activation in shared memory; every lane of the warp calls
__device__ __noinline__ void put_act(int type, unsigned char * xs, int c8, bool valid, float v0, float v1, float v2, float v3, float v4, float v5, float v6, float v7) {
    if (type == PI_TYPE_F16) {
        const __half2 h0 = __floats2half2_rn(v0, v1), h1 = __floats2half2_rn(v2, v3), h2 = __floats2half2_rn(v4, v5), h3 = __floats2half2_rn(v6, v7);
        if (valid) reinterpret_cast<uint4 *>(xs)[c8] = make_uint4(*reinterpret_cast<const uint32_t *>(&h0), *reinterpret_cast<const uint32_t *>(&h1),
                                                                  *reinterpret_cast<const uint32_t *>(&h2), *reinterpret_cast<const uint32_t *>(&h3));
        return;
    }
    const int nb = s_p.d / QK;                                        // quantize_row_q8_0, as emit_act8
    float amax = fmaxf(fmaxf(fmaxf(fabsf(v0), fabsf(v1)), fmaxf(fabsf(v2), fabsf(v3))), fmaxf(fmaxf(fabsf(v4), fabsf(v5)), fmaxf(fabsf(v6), fabsf(v7))));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    const float d = amax / 127.0f, id = amax != 0.0f ? 127.0f / amax : 0.0f;
    const int q0 = __float2int_rn(v0 * id), q1 = __float2int_rn(v1 * id), q2 = __float2int_rn(v2 * id), q3 = __float2int_rn(v3 * id);
    const int q4 = __float2int_rn(v4 * id), q5 = __float2int_rn(v5 * id), q6 = __float2int_rn(v6 * id), q7 = __float2int_rn(v7 * id);
    int s = q0 + q1 + q2 + q3 + q4 + q5 + q6 + q7;
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    const uint2 w = make_uint2(__byte_perm(__byte_perm(q0, q1, 0x0040), __byte_perm(q2, q3, 0x0040), 0x5410), __byte_perm(__byte_perm(q4, q5, 0x0040), __byte_perm(q6, q7, 0x0040), 0x5410));
    if (!valid) return;
    const int blk = c8 >> 2, part = c8 & 3;
    reinterpret_cast<uint2 *>(xs + ((part < 2 ? 0 : nb) + blk) * 16)[part & 1] = w;
    if (part == 0) reinterpret_cast<uint2 *>(xs + nb * 32)[blk] = make_uint2(__float_as_uint(__half2float(__float2half_rn(d))), (unsigned)s);
}

__device__ __noinline__ double sum_ct(double v) {
    v = warp_sum_d(v);
    bar_ct();                                                        // s_dred may still be read from the call before
    if ((threadIdx.x & 31) == 0) s_dred[threadIdx.x >> 5] = v;
    bar_ct();
    double t = 0.0;
    for (int i = 0; i < ST_WARPS; i++) t += s_dred[i];
    return t;
}

__device__ __forceinline__ void put_raw(unsigned char * xs, int c8, const float (&v)[8]) { put_act(PI_TYPE_F16, xs, c8, true, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]); }

// what a norm makes of its vector: planes of type `type` (weights w, bias b) in out, those of a second norm of the same vector in out2
// (when given), the vector itself in FP16 in raw (when given)
struct NormOut { const float * w, * b; unsigned char * out; const float * w2, * b2; unsigned char * out2, * raw; int type; };

// The norm of the vector behind `src` (numerics of k_norm), by every CTA for itself.
template <int NC>                                                     // groups of 8 values per thread
__device__ __noinline__ void norm_phase(const u64 * src, unsigned tag, const NormOut o) {
    const int tid = threadIdx.x, n = s_p.d;
    float v[NC][8];
#pragma unroll
    for (int k0 = 0; k0 < NC; k0 += 2) {
        u64 r[2][8];
        const int c = (k0 * ST_CT + tid) * 8;
        int polls = 0;
        while (true) {
            unsigned off = 0u;
#pragma unroll
            for (int k = 0; k < 2; k++)
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    r[k][j] = r[k][j + 1] = 0ull;
                    if (c + k * ST_CT * 8 < n) {
                        ld2(src + c + k * ST_CT * 8 + j, r[k][j], r[k][j + 1]);
                        off |= ((unsigned)(r[k][j] >> 32) ^ tag) | ((unsigned)(r[k][j + 1] >> 32) ^ tag);
                    }
                }
            if (!off || wait_over(polls)) break;
            // every CTA polls this vector: where it is more than a word pair a thread, one word until it is there (8 layers of d 8192: 603
            // us, 617 without; 12 layers of d 4096: 743 us with it, 726 without)
            if (n > ST_CT * 8) wait_words(src + c, 1, tag);
        }
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
            for (int j = 0; j < 8; j++) v[k0 + k][j] = val(r[k][j]);
    }
    float scale;
    if (s_p.rms) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < NC; k++)
#pragma unroll
            for (int j = 0; j < 8; j++) s += (double)(v[k][j] * v[k][j]);
        scale = 1.0f / sqrtf((float)(sum_ct(s) / (double)n) + s_p.eps);
    } else {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < NC; k++)
#pragma unroll
            for (int j = 0; j < 8; j++) s += (double)v[k][j];
        const float mean = (float)(sum_ct(s) / (double)n);
        s = 0.0;
#pragma unroll
        for (int k = 0; k < NC; k++)
            if ((k * ST_CT + tid) * 8 < n) {
                if (o.raw) put_raw(o.raw, k * ST_CT + tid, v[k]);
#pragma unroll
                for (int j = 0; j < 8; j++) { v[k][j] = v[k][j] - mean; s += (double)(v[k][j] * v[k][j]); }
            }
        scale = 1.0f / sqrtf((float)(sum_ct(s) / (double)n) + s_p.eps);
    }
#pragma unroll
    for (int k = 0; k < NC; k++) {
        if (k * ST_CT * 8 >= n) break;
        const int c8 = k * ST_CT + tid;
        const bool ok = c8 * 8 < n;
        if (ok && o.raw && s_p.rms) put_raw(o.raw, c8, v[k]);
#pragma unroll 1
        for (int t = 0; t < (o.out2 ? 2 : 1); t++) {
            const float * w = t ? o.w2 : o.w, * b = t ? o.b2 : o.b;
            float y[8];
#pragma unroll
            for (int j = 0; j < 8; j++) y[j] = __fmul_rn(v[k][j], scale);            // separate roundings, as separate graph nodes give
            if (ok && w) {
                const float4 p = __ldg(reinterpret_cast<const float4 *>(w) + 2 * c8), q = __ldg(reinterpret_cast<const float4 *>(w) + 2 * c8 + 1);
                y[0] = __fmul_rn(y[0], p.x); y[1] = __fmul_rn(y[1], p.y); y[2] = __fmul_rn(y[2], p.z); y[3] = __fmul_rn(y[3], p.w);
                y[4] = __fmul_rn(y[4], q.x); y[5] = __fmul_rn(y[5], q.y); y[6] = __fmul_rn(y[6], q.z); y[7] = __fmul_rn(y[7], q.w);
            }
            if (ok && b) {
                const float4 p = __ldg(reinterpret_cast<const float4 *>(b) + 2 * c8), q = __ldg(reinterpret_cast<const float4 *>(b) + 2 * c8 + 1);
                y[0] = __fadd_rn(y[0], p.x); y[1] = __fadd_rn(y[1], p.y); y[2] = __fadd_rn(y[2], p.z); y[3] = __fadd_rn(y[3], p.w);
                y[4] = __fadd_rn(y[4], q.x); y[5] = __fadd_rn(y[5], q.y); y[6] = __fadd_rn(y[6], q.z); y[7] = __fadd_rn(y[7], q.w);
            }
            put_act(o.type, t ? o.out2 : o.out, c8, ok, y[0], y[1], y[2], y[3], y[4], y[5], y[6], y[7]);
        }
    }
    bar_ct();
}

// the vector behind 4-byte words {16 bits, 16 bits of the number} as staged activation: FP16 values ...
__device__ __noinline__ void stage_f16(const uint32_t * src, int n, unsigned tag, unsigned char * xs) {
    tag <<= 16;
    constexpr int U = 4;
#pragma unroll 1
    for (int g0 = threadIdx.x; g0 < n / 4; g0 += ST_CT * U) {
        uint4 v[U];
#pragma unroll
        for (int u = 0; u < U; u++) if (g0 + u * ST_CT < n / 4) v[u] = ld4(src + (g0 + u * ST_CT) * 4);
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int g = g0 + u * ST_CT;
            if (g >= n / 4) break;
            if (((v[u].x ^ tag) | (v[u].y ^ tag) | (v[u].z ^ tag) | (v[u].w ^ tag)) >> 16) v[u] = wait_words4(src + g * 4, 16, tag);
            reinterpret_cast<uint2 *>(xs)[g] = make_uint2(__byte_perm(v[u].x, v[u].y, 0x5410), __byte_perm(v[u].z, v[u].w, 0x5410));
        }
    }
    bar_ct();
}
// ... or Q8_0 as int8 pairs and scales
__device__ __noinline__ void stage_q8(const uint32_t * src, const uint32_t * scales, int n, unsigned tag, unsigned char * xs) {
    const int ng = n / 8, nb = n / QK;                                 // 8 values a thread; four lanes share a block
    tag <<= 16;
    constexpr int U = 2;
#pragma unroll 1
    for (int g0 = 0; g0 < ng; g0 += ST_CT * U) {
        uint4 v[U];
        uint32_t sc[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int g = g0 + u * ST_CT + threadIdx.x;
            v[u] = make_uint4(tag, tag, tag, tag); sc[u] = tag;
            if (g < ng) { v[u] = ld4(src + g * 4); sc[u] = ldw(scales + (g >> 2)); }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int g = g0 + u * ST_CT + threadIdx.x;
            if (((v[u].x ^ tag) | (v[u].y ^ tag) | (v[u].z ^ tag) | (v[u].w ^ tag)) >> 16) v[u] = wait_words4(src + g * 4, 16, tag);
            if ((sc[u] ^ tag) >> 16) { wait_words4(scales + ((g >> 2) & ~3), 16, tag); sc[u] = ldw(scales + (g >> 2)); }
            const uint2 w = make_uint2(__byte_perm(v[u].x, v[u].y, 0x5410), __byte_perm(v[u].z, v[u].w, 0x5410));
            int s = __dp4a((int)w.x, 0x01010101, 0);
            s = __dp4a((int)w.y, 0x01010101, s);
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            if (g < ng) {
                const int blk = g >> 2, part = g & 3;
                reinterpret_cast<uint2 *>(xs + ((part < 2 ? 0 : nb) + blk) * 16)[part & 1] = w;
                if (part == 0) reinterpret_cast<uint2 *>(xs + nb * 32)[blk] = make_uint2(__float_as_uint(__half2float(__ushort_as_half((unsigned short)(sc[u] & 0xffffu)))), (unsigned)s);
            }
        }
    }
    bar_ct();
}

// ------------------------------------------------------------------------------------------------ attention of one head

// k_attention_row with its inputs and outputs as words that carry their own validity (same arithmetic, same order)
template <int HC>
__device__ __noinline__ void attention_head(int h, int layer, int pos, int seq, unsigned tag) {
    struct { int n_ctx, n_head, n_head_kv, max_batch, dq, dkv, neox, q4; const float * cs; } p;
    p.n_ctx = s_p.n_ctx; p.n_head = s_p.n_head; p.n_head_kv = s_p.n_head_kv; p.max_batch = s_p.max_batch; p.dq = s_p.dq; p.dkv = s_p.dkv; p.neox = s_p.neox; p.q4 = s_p.q4; p.cs = s_p.cs;
    const u64 * qkv = s_p.qkv + (size_t)(layer & 1) * (p.dq + 2 * p.dkv);
    unsigned char * scratch = smem + s_p.off_b;
    constexpr int HD = HC * 32, HALF = HD / 2, CH = HD / 8, SL = ST_CT / CH, NW = ST_WARPS;
    constexpr int UV = 6;                                             // value rows of a thread on their way
    float * red = reinterpret_cast<float *>(scratch);                 // [NW][HD]
    __half * q16 = reinterpret_cast<__half *>(red + NW * HD);
    __half * k16 = q16 + HD;
    __half * v16 = k16 + HD;
    unsigned * s_sum = reinterpret_cast<unsigned *>(v16 + HD);
    int * s_max = reinterpret_cast<int *>(s_sum + NW);
    float * sc = reinterpret_cast<float *>(s_max + NW);               // [n_ctx] scores
    __half * p16 = reinterpret_cast<__half *>(sc + p.n_ctx);          // [n_ctx] probabilities
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, g = lane >> 2, q = lane & 3;
    const int group = p.n_head / p.n_head_kv, hk = h / group, dkv = p.n_head_kv * HD;
    const size_t off = ((size_t)layer * p.max_batch + seq) * p.n_ctx * dkv + (size_t)hk * HD;
    __half * kc = s_p.k_cache + off;
    __half * vc = s_p.v_cache + off;
    const bool inside = pos >= 0 && pos < p.n_ctx;                    // never index the cache out of range
    if (!inside) pos = 0;
    // ---- before the query is there: earlier steps stored these rows
    uint4 kv[2][HC];
    auto keys = [&](int j0) {
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int c = 0; c < HC; c++) kv[r][c] = j0 + g + 8 * r < pos ? *(reinterpret_cast<const uint4 *>(kc + (size_t)(j0 + g + 8 * r) * dkv) + c * 4 + q) : make_uint4(0u, 0u, 0u, 0u);
    };
    keys(wid * 16);
#pragma unroll 1
    for (int j = tid; j < pos; j += ST_CT) {
        const char * vr = reinterpret_cast<const char *>(vc + (size_t)j * dkv);
#pragma unroll
        for (int o = 0; o < HD * 2; o += 128) asm volatile("prefetch.global.L2 [%0];" :: "l"(vr + o));
    }
    // ---- the query and the new key, rotated, and the new value, as FP16
    if (tid < HD) {
        const int t = tid < HALF ? tid : tid - HALF;
        float2 cs = make_float2(1.f, 0.f);
        if (p.cs) cs = reinterpret_cast<const float2 *>(p.cs)[(size_t)pos * HALF + t];
        const u64 * s = tid < HALF ? qkv + (size_t)h * HD : qkv + p.dq + (size_t)hk * HD;
        const int i0 = p.cs && !p.neox ? 2 * t : t, i1 = p.cs && !p.neox ? 2 * t + 1 : t + HALF;
        u64 x0 = ld1(s + i0), x1 = ld1(s + i1);
        if (!fresh(x0, tag)) x0 = wait_words(s + i0, 1, tag);
        if (!fresh(x1, tag)) x1 = wait_words(s + i1, 1, tag);
        float a0 = val(x0), a1 = val(x1);
        if (p.cs) { float o0, o1; rope_pair(a0, a1, cs.x, cs.y, o0, o1); a0 = o0; a1 = o1; }
        __half * d16 = tid < HALF ? q16 : k16;
        d16[i0] = __float2half_rn(a0); d16[i1] = __float2half_rn(a1);
    } else if (tid >= 256 && tid < 256 + HD) {
        v16[tid - 256] = __float2half_rn(wait_val(qkv + p.dq + p.dkv + (size_t)hk * HD + tid - 256, tag));
    }
    bar_ct();
    if (h % group == 0 && tid < HD && inside) {
        kc[(size_t)pos * dkv + tid] = k16[tid];
        vc[(size_t)pos * dkv + tid] = v16[tid];
    }
    // ---- scores
    const float scale = 1.0f / sqrtf((float)HD);
    uint4 bq[HC];
#pragma unroll
    for (int c = 0; c < HC; c++) bq[c] = *(reinterpret_cast<const uint4 *>(q16) + c * 4 + q);
    float mx = -INFINITY;
    auto mma = [&](float (&c4)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(c4[0]), "+f"(c4[1]), "+f"(c4[2]), "+f"(c4[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    };
#pragma unroll 1
    for (int j0 = wid * 16; j0 <= pos; j0 += NW * 16) {               // rows j0 .. j0 + 15, of which this lane holds g and g + 8
#pragma unroll
        for (int r = 0; r < 2; r++)
            if (j0 + g + 8 * r == pos) {
#pragma unroll
                for (int c = 0; c < HC; c++) kv[r][c] = *(reinterpret_cast<const uint4 *>(k16) + c * 4 + q);
            }
        __syncwarp();
        float x[4] = {0.f, 0.f, 0.f, 0.f}, y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < HC; c++) {
            mma(x, kv[0][c].x, kv[1][c].x, kv[0][c].y, kv[1][c].y, bq[c].x, bq[c].y);
            mma(y, kv[0][c].z, kv[1][c].z, kv[0][c].w, kv[1][c].w, bq[c].z, bq[c].w);
        }
        keys(j0 + NW * 16);
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const int j = j0 + g + 8 * r;
            const float s = (x[2 * r] + y[2 * r]) * scale;
            if (j <= pos) { mx = fmaxf(mx, s); if (q == 0) sc[j] = s; }
        }
    }
    // ---- the first value rows of this thread: 8 columns c8 of rows sl, sl + SL, ...
    const int c8 = tid % CH, sl = tid / CH;
    uint4 vv[UV];
    auto values = [&](int j0) {
#pragma unroll
        for (int u = 0; u < UV; u++) {
            const int j = j0 + u * SL;
            vv[u] = make_uint4(0u, 0u, 0u, 0u);
            if (j < pos) vv[u] = *(reinterpret_cast<const uint4 *>(vc + (size_t)j * dkv) + c8);
            else if (j == pos) vv[u] = reinterpret_cast<const uint4 *>(v16)[c8];
        }
    };
    values(sl);
    auto ordered = [](int b) { return b ^ ((b >> 31) & 0x7fffffff); };
    const int mi = __reduce_max_sync(0xffffffffu, ordered(__float_as_int(mx)));
    if (lane == 0) s_max[wid] = mi;
    bar_ct();
    int m = s_max[0];
#pragma unroll 5
    for (int i = 1; i < NW; i++) m = max(m, s_max[i]);
    mx = __int_as_float(ordered(m));
    // ---- softmax (ggml.c:10708-10777)
    unsigned part = 0u;
#pragma unroll 1
    for (int j = tid; j <= pos; j += ST_CT) {
        const float e = round_f16(expf(round_f16(sc[j] - mx)));
        sc[j] = e;
        part += (unsigned)(e * 16777216.0f);                          // exact; 2^24 at most, for up to 7 positions of a thread (step_plan)
    }
    const unsigned ws = __reduce_add_sync(0xffffffffu, part);
    if (lane == 0) s_sum[wid] = ws;
    bar_ct();
    {
        unsigned long long tot = 0ull;
#pragma unroll
        for (int i = 0; i < NW; i++) tot += s_sum[i];
        const float inv = (float)(1.0 / ((double)tot * (1.0 / 16777216.0)));
#pragma unroll 1
        for (int j = tid; j <= pos; j += ST_CT) p16[j] = __float2half_rn(sc[j] * inv);
    }
    bar_ct();
    // ---- out[e] = sum_j p_j V[j, e]
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int j0 = sl; j0 <= pos; j0 += SL * UV) {
        if (j0 != sl) values(j0);
#pragma unroll
        for (int u = 0; u < UV; u++) {
            const int j = j0 + u * SL;
            const uint4 v = vv[u];
            const float pj = j <= pos ? __half2float(p16[j]) : 0.f;
            const float2 v0 = h2f(v.x), v1 = h2f(v.y), v2 = h2f(v.z), v3 = h2f(v.w);
            acc[0] = fmaf(pj, v0.x, acc[0]); acc[1] = fmaf(pj, v0.y, acc[1]); acc[2] = fmaf(pj, v1.x, acc[2]); acc[3] = fmaf(pj, v1.y, acc[3]);
            acc[4] = fmaf(pj, v2.x, acc[4]); acc[5] = fmaf(pj, v2.y, acc[5]); acc[6] = fmaf(pj, v3.x, acc[6]); acc[7] = fmaf(pj, v3.y, acc[7]);
        }
    }
    __syncwarp();
#pragma unroll
    for (int o = CH; o < 32; o <<= 1)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
    if (lane < CH) {
        *reinterpret_cast<float4 *>(red + wid * HD + lane * 8) = make_float4(acc[0], acc[1], acc[2], acc[3]);
        *reinterpret_cast<float4 *>(red + wid * HD + lane * 8 + 4) = make_float4(acc[4], acc[5], acc[6], acc[7]);
    }
    bar_ct();
    if (tid < HD) {
        float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int w = 0; w < NW; w++) o[w & 3] += red[w * HD + tid];
        const float v = (o[0] + o[1]) + (o[2] + o[3]);
        const int e = h * HD + tid;
        uint32_t * out = s_p.acto + (size_t)(layer & 1) * p.dq, * out_scale = s_p.acts + (size_t)(layer & 1) * (p.dq / QK);
        if (!p.q4) {
            stw(out + e, (tag << 16) | __half_as_ushort(__float2half_rn(v)));
        } else {                                                      // quantize_row_q8_0, a block per warp; two int8 per word
            const float amax = warp_max(fabsf(v));
            const float d = amax / 127.0f, id = amax != 0.0f ? 127.0f / amax : 0.0f;
            const int qv = __float2int_rn(v * id), other = __shfl_down_sync(0xffffffffu, qv, 1);
            if ((lane & 1) == 0) stw(out + e / 2, (tag << 16) | (uint32_t)(qv & 0xff) | ((uint32_t)(other & 0xff) << 8));
            if (lane == 0) stw(out_scale + e / QK, (tag << 16) | __half_as_ushort(__float2half_rn(d)));
        }
    }
    bar_ct();                                                         // the scratch is free again
}

// ------------------------------------------------------------------------------------------------ the sparse FFN

// the predictor's masks -> sh_mask, sh_pref (exclusive prefix of the counts); returns the number of active rows
__device__ __noinline__ int scan_words(const uint32_t * src, unsigned tag) {
    uint32_t * s_mask = sh_mask();
    int * s_pref = sh_pref();
    const int wpt = s_p.wpt, F = s_p.F;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, n_chunks = F / 32;
    tag <<= 8;
    uint32_t m[4] = {0u, 0u, 0u, 0u};
    uint4 v[4];
    const int c0 = tid * wpt;
#pragma unroll
    for (int k = 0; k < 4; k++) if (k < wpt && c0 + k < n_chunks) v[k] = ld4(src + (c0 + k) * 4);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (k >= wpt || c0 + k >= n_chunks) continue;
        if (((v[k].x ^ tag) | (v[k].y ^ tag) | (v[k].z ^ tag) | (v[k].w ^ tag)) >> 8) v[k] = wait_words4(src + (c0 + k) * 4, 8, tag);
        m[k] = __byte_perm(__byte_perm(v[k].x, v[k].y, 0x0040), __byte_perm(v[k].z, v[k].w, 0x0040), 0x5410);
    }
    int mine = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) mine += __popc(m[k]);
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += x;
    }
    if (lane == 31) s_warp[wid] = incl;
    bar_ct();
    int base = 0;
#pragma unroll 4
    for (int w = 0; w < wid; w++) base += s_warp[w];
    int off = base + incl - mine;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (k < wpt && c0 + k < n_chunks) { s_mask[c0 + k] = m[k]; s_pref[c0 + k] = off; off += __popc(m[k]); }
    }
    if (tid == ST_CT - 1) s_pref[n_chunks] = base + incl;
    bar_ct();
    return s_pref[n_chunks];
}

// the rows whose ranks lie in [lo, hi) into dst[rank - lo]; every thread expands the words it owns
__device__ __forceinline__ void list_rows(int lo, int hi, int * dst) {
    const uint32_t * s_mask = sh_mask();
    const int * s_pref = sh_pref();
    const int n_chunks = s_p.F / 32, wpt = s_p.wpt;
    const int c0 = min((int)threadIdx.x * wpt, n_chunks), c1 = min(c0 + wpt, n_chunks);
#pragma unroll 1
    for (int k = c0; k < c1; k++) {
        int rank = s_pref[k];
        uint32_t mk = s_mask[k];
        if (rank >= hi || rank + __popc(mk) <= lo) continue;
#pragma unroll 1
        while (mk) {
            const int bit = __ffs(mk) - 1;
            mk &= mk - 1;
            if (rank >= lo && rank < hi) dst[rank - lo] = k * 32 + bit;
            rank++;
        }
    }
}

// this CTA's rows of the gather, by rank: listed for the copying warps
template <bool GATED>
__device__ __forceinline__ void gather_list(int layer, int n) {
    if (layer) wait_bar(&s_taken, (unsigned)(layer - 1) & 1u);
    const int first = (int)(blockIdx.x * (unsigned)n / gridDim.x), mj = (int)((blockIdx.x + 1) * (unsigned)n / gridDim.x) - first;
    list_rows(first, first + mj, sh_rows());
    if (threadIdx.x == 0) {
        s_rows[ST_GATHER] = GATED ? 2 * mj : mj;
        s_slots[ST_GATHER] = mat_slots(s_p.mat[ST_GATHER], GATED ? 2 * mj : mj);
        s_gather = (unsigned)s_rows[ST_GATHER] | (unsigned)s_slots[ST_GATHER] << 16;
        s_kb = s_p.F / 32; s_ke = s_p.F / 32;                         // (axpy_phase looks for its range)
    }
    bar_ct();
    if (threadIdx.x == 0) mbar_arrive(&s_listed);
}

// h = relu(gate . x) * (up . x) | relu(up . x + b) over the rows of this CTA; an up row and its gate row follow one another in the ring
template <int WT, bool GATED>
__device__ __noinline__ void gather_phase(int layer, unsigned kbase, unsigned tag) {
    constexpr int NM = GATED ? 2 : 1;
    const int n = s_rows[ST_GATHER], chunk = s_p.mat[ST_GATHER].chunk;   // (an even number of rows)
    const int * rows = sh_rows();
    const float * bias = s_layer[layer & 1].f[ST_BUP];
    u64 * out = s_p.h + (size_t)(layer & 1) * s_p.F;
#pragma unroll 1
    for (int c0 = 0; c0 < n; c0 += chunk) {
        const int nc = min(chunk, n - c0);
        consume<WT>(ST_GATHER, kbase + slot_of(ST_GATHER, c0), nc, smem + s_p.off_a);
#pragma unroll 1
        for (int t = threadIdx.x; t < nc / NM; t += ST_CT) {
            const int r = rows[c0 / NM + t];
            float o = row_total(ST_GATHER, t * NM);
            if (GATED) o = fmaxf(row_total(ST_GATHER, t * NM + 1), 0.f) * o;
            if (bias) o += bias[r];
            if (s_p.relu) o = fmaxf(o, 0.f);
            st1(out + r, o, tag);
        }
        bar_ct();
    }
}

// one CTA's share of the axpy: a slice of 1024 columns, the rows of a group of whole mask words
template <int WT>
__device__ __noinline__ void axpy_phase(int layer, int n, unsigned tag) {
    constexpr int UA = WT == PI_TYPE_F16 ? 4 : 8;                     // rows in flight per warp (half as many: 568 instead of 554 us for 4 layers of the 40B shape)
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nb = s_p.d / QK, n_chunks = s_p.F / 32, wpt = s_p.wpt;
    const int units = WT == PI_TYPE_F16 ? s_p.d / 8 : nb;
    const int n_slices = (s_p.d + SLICE - 1) / SLICE, slice = blockIdx.x % n_slices, group = blockIdx.x / n_slices;
    if (group >= s_p.groups) return;
    const int unit0 = WT == PI_TYPE_F16 ? slice * (SLICE / 8) + lane : slice * 32 + lane;
    const uint8_t * Wdown = s_layer[layer & 1].w[ST_DOWN];
    const int64_t row_bytes = s_p.row_bytes;
    const uint32_t * s_mask = sh_mask();
    const int * s_pref = sh_pref();
    int * s_row = sh_list();
    float * s_h = reinterpret_cast<float *>(s_row + ST_LIST);
    int * s_row2 = s_row + 2 * ST_LIST;
    float * s_coef = s_h + 2 * ST_LIST;
    {
        // the group's range of mask words: from the first word at which the running count reaches the group's share
        const int tb = (int)((unsigned)group * (unsigned)n / (unsigned)s_p.groups), te = (int)((unsigned)(group + 1) * (unsigned)n / (unsigned)s_p.groups);
        const bool last = group + 1 >= s_p.groups;
        const int c0 = min(tid * wpt, n_chunks), c1 = min(c0 + wpt, n_chunks);
        for (int k = c0; k < c1; k++) {
            const int here = s_pref[k];
            if (here >= tb && (k == 0 || s_pref[k - 1] < tb)) s_kb = k;
            if (!last && here >= te && (k == 0 || s_pref[k - 1] < te)) s_ke = k;
        }
        bar_ct();
    }
    const int kb = s_kb, ke = s_ke;
    u64 acc[16];
    float corr = 0.f;
#pragma unroll
    for (int j = 0; j < 16; j++) acc[j] = 0ull;
#pragma unroll 1
    for (int ka = kb; ka < ke;) {
        // as many whole words as hold at most ST_LIST rows
        int kz = ke;
        if (s_pref[ke] - s_pref[ka] > ST_LIST) {
            const int c0 = max(min(tid * wpt, n_chunks), ka + 1), c1 = min(min(tid * wpt + wpt, n_chunks), ke);
            for (int k = c0; k < c1; k++)
                if (s_pref[k] - s_pref[ka] <= ST_LIST && s_pref[k + 1] - s_pref[ka] > ST_LIST) s_kz = k;
            bar_ct();
            kz = s_kz;
        }
        const int r0 = s_pref[ka], m = s_pref[kz] - r0;
        list_rows(r0, r0 + m, s_row);
        bar_ct();
        int r = -1;
        float c = 0.f;
        if (tid < m) {
            r = s_row[tid];
            c = wait_val(s_p.h + (size_t)(layer & 1) * s_p.F + r, tag);
            s_h[tid] = c;
        }
        if (WT == PI_TYPE_F16) {
            c = round_f16(c);
        } else {
            // the int8 quant of h within its block of 32 neurons times that block's FP16 scale (quantize_row_q8_0); inactive
            // neurons of the block count as 0, and the active ones are neighbours in rank order
            bar_ct();
            if (tid < m) {
                const int ch = r >> 5, f = s_pref[ch] - r0, cnt = __popc(s_mask[ch]);
                float amax = 0.f;
#pragma unroll 4
                for (int i = 0; i < cnt; i++) amax = fmaxf(amax, fabsf(s_h[f + i]));
                const float id = amax != 0.0f ? 127.0f / amax : 0.0f;
                c = (float)__float2int_rn(c * id) * round_f16(amax / 127.0f);
            }
        }
        // rows whose coefficient is not zero (the CPU path skips the others too: ggml.c:14422-14428, 14571-14581), in order
        const bool keep = r >= 0 && c != 0.f;
        const unsigned bal = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) s_warp[wid] = __popc(bal);
        bar_ct();
        int off = 0, m2 = 0;
#pragma unroll 4
        for (int w = 0; w < ST_WARPS; w++) { const int c16 = s_warp[w]; if (w < wid) off += c16; m2 += c16; }
        if (keep) { const int o = off + __popc(bal & ((1u << lane) - 1u)); s_row2[o] = r; s_coef[o] = c; }
        bar_ct();
        // warp w takes entries w, w + 16, ...; a lane owns 32 columns of the slice:
        //   Q4_0: block `slice * 32 + lane` (sum index = column inside the block);
        //   FP16: 8 columns at 8 * lane of each of the slice's four 256-column quarters (sum index = 8 * quarter + e)
#pragma unroll 1
        for (int e0 = wid; e0 < m2; e0 += ST_WARPS * UA) {
            if (WT == PI_TYPE_Q4_0) {
                uint4 q[UA]; __half d4[UA]; float cf[UA];
#pragma unroll
                for (int u = 0; u < UA; u++) {
                    const int i = e0 + u * ST_WARPS;
                    cf[u] = 0.f; q[u] = make_uint4(0u, 0u, 0u, 0u); d4[u] = __ushort_as_half((unsigned short)0);
                    if (i < m2) {
                        cf[u] = s_coef[i];
                        const uint8_t * row = Wdown + (size_t)s_row2[i] * row_bytes;
                        if (unit0 < units) {
                            q[u] = ldg_stream(reinterpret_cast<const uint4 *>(row) + unit0);
                            d4[u] = __ldg(reinterpret_cast<const __half *>(row + (size_t)nb * 16) + unit0);
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < UA; u++) {
                    // nibble q -> the float 16 + q with one byte permute; (q - 8) * sc = (16 + q) * sc - 24 * sc (see k_ffn_rows)
                    const float sc = cf[u] * __half2float(d4[u]);
                    corr += sc;
                    const u64 sc2 = pack2(sc, sc);
                    const uint32_t wds[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
#pragma unroll
                    for (int wi = 0; wi < 4; wi++) {
                        const uint32_t lo = ((wds[wi] << 3) & 0x78787878u) | 0x80808080u;
                        const uint32_t hi = ((wds[wi] >> 1) & 0x78787878u) | 0x80808080u;
                        const u64 l01 = (u64)__byte_perm(lo, 0x41000000u, 0x7044u) | ((u64)__byte_perm(lo, 0x41000000u, 0x7144u) << 32);
                        const u64 l23 = (u64)__byte_perm(lo, 0x41000000u, 0x7244u) | ((u64)__byte_perm(lo, 0x41000000u, 0x7344u) << 32);
                        const u64 h01 = (u64)__byte_perm(hi, 0x41000000u, 0x7044u) | ((u64)__byte_perm(hi, 0x41000000u, 0x7144u) << 32);
                        const u64 h23 = (u64)__byte_perm(hi, 0x41000000u, 0x7244u) | ((u64)__byte_perm(hi, 0x41000000u, 0x7344u) << 32);
                        ffma2(acc[wi * 2], l01, sc2); ffma2(acc[wi * 2 + 1], l23, sc2);
                        ffma2(acc[8 + wi * 2], h01, sc2); ffma2(acc[8 + wi * 2 + 1], h23, sc2);
                    }
                }
            } else {
                uint4 w[UA][4]; float cf[UA];
#pragma unroll
                for (int u = 0; u < UA; u++) {
                    const int i = e0 + u * ST_WARPS;
                    cf[u] = i < m2 ? s_coef[i] : 0.f;
                    const uint4 * row = i < m2 ? reinterpret_cast<const uint4 *>(Wdown + (size_t)s_row2[i] * row_bytes) : nullptr;
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        w[u][k] = make_uint4(0u, 0u, 0u, 0u);
                        if (i < m2 && unit0 + k * 32 < units) w[u][k] = ldg_stream(row + unit0 + k * 32);
                    }
                }
#pragma unroll
                for (int u = 0; u < UA; u++) {
                    const u64 c2 = pack2(cf[u], cf[u]);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const float2 f0 = h2f(w[u][k].x), f1 = h2f(w[u][k].y), f2 = h2f(w[u][k].z), f3 = h2f(w[u][k].w);
                        ffma2(acc[k * 4 + 0], pack2(f0.x, f0.y), c2); ffma2(acc[k * 4 + 1], pack2(f1.x, f1.y), c2);
                        ffma2(acc[k * 4 + 2], pack2(f2.x, f2.y), c2); ffma2(acc[k * 4 + 3], pack2(f3.x, f3.y), c2);
                    }
                }
            }
        }
        if (kz < ke) bar_ct();                                       // the lists are written again
        ka = kz;
    }
    // ---- the warps' sums (index a of lane l at a * 33 + l: no bank conflicts), eight warps at a time, added in warp order
    float * s_red = reinterpret_cast<float *>(smem + s_p.off_a);
    float v0 = 0.f, v1 = 0.f;                                         // columns tid and tid + 512 of the slice
    int at0, at1;
    if (WT == PI_TYPE_Q4_0) { at0 = (tid & 31) * 33 + (tid >> 5); at1 = at0 + 16; }
    else                    { at0 = ((tid >> 8) * 8 + (tid & 7)) * 33 + ((tid & 255) >> 3); at1 = at0 + 16 * 33; }
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
        bar_ct();                                                     // what was in this place is dead for every warp
        if (wid >> 3 == half) {
            float * mine = s_red + (wid & 7) * (32 * 33) + lane;
#pragma unroll
            for (int j = 0; j < 16; j++) {
                float a = lo_f(acc[j]), b = hi_f(acc[j]);
                if (WT == PI_TYPE_Q4_0) { a = fmaf(-24.0f, corr, a); b = fmaf(-24.0f, corr, b); }
                mine[(2 * j) * 33] = a; mine[(2 * j + 1) * 33] = b;
            }
        }
        bar_ct();
#pragma unroll 4
        for (int w = 0; w < 8; w++) { v0 += s_red[w * (32 * 33) + at0]; v1 += s_red[w * (32 * 33) + at1]; }
    }
    u64 * out = s_p.part + ((size_t)(layer & 1) * s_p.groups + group) * s_p.d + slice * SLICE;
    const int left = s_p.d - slice * SLICE;
    if (tid < left) st1(out + tid, v0, tag);
    if (tid + ST_CT < left) st1(out + tid + ST_CT, v1, tag);
}

// ------------------------------------------------------------------------------------------------ the dense nodes of a layer

__device__ __forceinline__ void norm_any(const u64 * src, unsigned tag, const NormOut & o) {
    if (s_p.d <= 2 * ST_CT * 8) norm_phase<2>(src, tag, o);
    else                        norm_phase<4>(src, tag, o);
}

template <int WT>
__device__ __noinline__ void qkv_phase(int layer, unsigned kbase, unsigned tag) {
    const StepLayer & L = s_layer[layer & 1];
    const float * bias = L.f[ST_BQKV] ? L.f[ST_BQKV] + s_first[ST_QKV] : nullptr;
    float b = 0.f;
    if (bias && threadIdx.x < s_rows[ST_QKV]) b = bias[threadIdx.x];
    u64 * out = s_p.qkv + (size_t)(layer & 1) * (s_p.dq + 2 * s_p.dkv) + s_first[ST_QKV];
    rows_of<WT>(ST_QKV, kbase, smem + (s_p.falcon && !L.f[ST_N2W] ? s_p.off_a : s_p.off_c), [&](int t, float o) {
        if (bias) o += t == threadIdx.x ? b : bias[t];
        st1(out + t, o, tag);
    });
}

// attention output projection (+ bias); llama, opt: + the residual
template <int WT>
__device__ __noinline__ void wo_phase(int layer, unsigned kbase, unsigned tag) {
    const StepLayer & L = s_layer[layer & 1];
    const int tid = threadIdx.x, n = s_rows[ST_WO], first = s_first[ST_WO], par = layer & 1;
    const float * bias = L.f[ST_BO] ? L.f[ST_BO] + first : nullptr;
    const u64 * x = s_p.falcon ? nullptr : s_p.x + (size_t)par * s_p.d + first;
    float b = 0.f, res = 0.f;
    if (tid < n) { if (bias) b = bias[tid]; if (x) res = val(ld1(x + tid)); }
    if (WT == PI_TYPE_F16) stage_f16(s_p.acto + (size_t)par * s_p.dq, s_p.dq, tag, smem + s_p.off_c);
    else                   stage_q8(s_p.acto + (size_t)par * s_p.dq, s_p.acts + (size_t)par * (s_p.dq / QK), s_p.dq, tag, smem + s_p.off_c);
    u64 * out = s_p.x2 + (size_t)par * s_p.d + first;
    rows_of<WT>(ST_WO, kbase, smem + s_p.off_c, [&](int t, float o) {
        if (bias) o += t == tid ? b : bias[t];
        if (x) o += t == tid ? res : val(ld1(x + t));
        st1(out + t, o, tag);
    });
}

// hidden = relu(fc1 . x), FP16 (llama.cpp:4688-4691)
__device__ __noinline__ void fc1_phase(int layer, unsigned kbase, unsigned tag) {
    uint32_t * out = s_p.hid + (size_t)(layer & 1) * s_p.rank + s_first[ST_FC1];
    rows_of<PI_TYPE_F16>(ST_FC1, kbase, smem + s_p.off_b, [&](int t, float o) { stw(out + t, (tag << 16) | __half_as_ushort(__float2half_rn(fmaxf(o, 0.f)))); });
}

// the predictor's logits and masks (llama.cpp:4692-4695)
__device__ __noinline__ void fc2_phase(int layer, unsigned kbase, unsigned tag) {
    stage_f16(s_p.hid + (size_t)(layer & 1) * s_p.rank, s_p.rank, tag, smem + s_p.off_h);
    const int n = s_rows[ST_FC2], first = s_first[ST_FC2], chunk = s_p.mat[ST_FC2].chunk;    // (chunks of whole groups of 8 rows)
    float * pred = s_p.pred + (size_t)layer * s_p.pred_stride + first;
    uint32_t * out = s_p.maskw + (size_t)(layer & 1) * (s_p.F / 8) + first / 8;
#pragma unroll 1
    for (int c0 = 0; c0 < n; c0 += chunk) {
        const int nc = min(chunk, n - c0);
        consume<PI_TYPE_F16>(ST_FC2, kbase + slot_of(ST_FC2, c0), nc, smem + s_p.off_h);
#pragma unroll 1
        for (int t0 = 0; t0 < nc; t0 += ST_CT) {
            const int t = t0 + threadIdx.x;
            float o = 0.f;
            if (t < nc) { o = row_total(ST_FC2, t); pred[c0 + t] = o; }
            const unsigned bal = __ballot_sync(0xffffffffu, t < nc && !(o < s_p.threshold));   // (a NaN counts as active)
            const int lane = threadIdx.x & 31;
            if ((lane & 7) == 0 && t < nc) stw(out + (c0 + t) / 8, (tag << 8) | ((bal >> lane) & 0xffu));
        }
        bar_ct();
    }
}

// this CTA's columns of the residual stream: the partial vectors in group order (+ bias), + attention (falcon), + residual
__device__ __noinline__ void reduce_phase(int layer, unsigned tag) {
    const int tid = threadIdx.x, lane = tid & 31, par = layer & 1, groups = s_p.groups, d = s_p.d, col0 = s_col0, ncol = s_ncol;
    float * s_part = sh_part();
    const float * bias = s_layer[par].f[ST_BDOWN];
    float res = 0.f, att = 0.f, b = 0.f;
    bar_ct();                                                         // s_part is written again
    if (tid < ncol) {
        if (bias) b = bias[col0 + tid];
        res = wait_val(s_p.x2 + (size_t)par * d + col0 + tid, tag);
        if (s_p.falcon) { att = res; res = val(ld1(s_p.x + (size_t)par * d + col0 + tid)); }
    }
    // a warp per group, a lane per pair of columns (ncol is a multiple of 8)
#pragma unroll 1
    for (int g = tid >> 5; g < groups; g += ST_WARPS) {
        const u64 * part = s_p.part + ((size_t)par * groups + g) * d + col0;
#pragma unroll 1
        for (int c = 2 * lane; c < ncol; c += 64) {
            u64 x, y;
            ld2(part + c, x, y);
            if (!fresh(x, tag) || !fresh(y, tag)) { wait_words(part + c, 2, tag); ld2(part + c, x, y); }
            s_part[g * ncol + c] = val(x); s_part[g * ncol + c + 1] = val(y);
        }
    }
    bar_ct();
    if (tid < ncol) {
        float v = 0.f;
#pragma unroll 4
        for (int g = 0; g < groups; g++) v += s_part[g * ncol + tid];
        if (bias) v += b;
        if (s_p.falcon) v += att;
        v += res;
        st1(s_p.x + (size_t)(par ^ 1) * d + col0 + tid, v, tag + 1u);
    }
}

// ggml_get_rows on the embedding (+ OPT's learned positions at pos + 2: llama.cpp:5105-5108): this CTA's columns
__device__ __noinline__ void embed_phase(int token, int pos, unsigned tag) {
    const int d = s_p.d, col0 = s_col0, ncol = s_ncol;
#pragma unroll 1
    for (int c = threadIdx.x; c < ncol; c += ST_CT) {
        const int tok = token < 0 ? 0 : (token >= s_p.n_vocab ? s_p.n_vocab - 1 : token);
        float v = __half2float(s_p.tok_embd[(size_t)tok * d + col0 + c]);
        if (s_p.pos_embd) {
            int q = pos + 2;
            q = q < 0 ? 0 : (q >= s_p.n_pos ? s_p.n_pos - 1 : q);
            v = v + __half2float(s_p.pos_embd[(size_t)q * d + col0 + c]);
        }
        st1(s_p.x + col0 + c, v, tag);
    }
}

// lm head and greedy choice (the first index of the maximum, as k_argmax)
template <int WT>
__device__ __noinline__ void head_phase(unsigned kbase) {
    const int tid = threadIdx.x, first = s_first[ST_HEAD];
    float * logits = s_p.logits + first, * host = s_p.logits_host ? s_p.logits_host + first : nullptr;
    u64 key = 0ull;
    auto done = [&](int t, float v) {
        logits[t] = v;
        if (host) host[t] = v;
        if (!(v > -INFINITY)) return;
        const unsigned b = __float_as_uint(v + 0.f);
        const u64 k = ((u64)(b >> 31 ? ~b : b | 0x80000000u) << 32) | ~(unsigned)(first + t);
        key = k > key ? k : key;
    };
    if (WT == PI_TYPE_Q4_0 && s_p.head_type == PI_TYPE_Q4_0) rows_of<PI_TYPE_Q4_0>(ST_HEAD, kbase, smem + s_p.off_a, done);
    else                                                     rows_of<PI_TYPE_F16>(ST_HEAD, kbase, smem + s_p.off_a, done);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { const u64 k = __shfl_xor_sync(0xffffffffu, key, o); key = k > key ? k : key; }
    u64 * s_key = reinterpret_cast<u64 *>(s_dred);
    if ((tid & 31) == 0) { s_key[tid >> 5] = key; mbar_arrive(&s_done); }
    bar_ct();
    if (tid != 0) return;
    if (atomicCAS(const_cast<int *>(&s_dead), 0, 2) == 1) end_step();  // (a copying warp has said so or is about to: the last CTA shall see it)
    for (int w = 1; w < ST_WARPS; w++) key = s_key[w] > key ? s_key[w] : key;
    if (key) atomicMax(s_p.best, key);
    __threadfence();
    if (atomicAdd(s_p.ticket, 1u) != gridDim.x - 1u) return;
    __threadfence();
    const u64 k = atomicExch(s_p.best, 0ull);
    const bool ended = ldw(s_p.abort) == s_step + 1u;
    *s_p.ticket = 0u;
    *s_p.step_no = s_step + 1u;                                       // every CTA has read it: all have taken a ticket
    const int32_t i = ended ? -1 : (k ? (int32_t)~(unsigned)k : 0);
    *s_p.argmax = i;
    if (s_p.argmax_host) *s_p.argmax_host = i;
}

// ------------------------------------------------------------------------------------------------ the copying warps: one lane of each

struct Copier { unsigned k, s, par, bs, bpar; };                     // this copier's next slot, its place, the round's parity; the slot `window` places back

// the slots of `nrow` rows from kbase on that are this copier's (k % ST_COPY == me); false: a wait ran out
template <bool GATED>
__device__ __noinline__ bool issue(int mi, const uint8_t * W, const uint8_t * W2, unsigned kbase, int nrow, int nslots, Copier & cp) {
    const int rps = s_p.mat[mi].rps, pieces = s_p.mat[mi].pieces, units = s_p.mat[mi].units, punits = s_p.mat[mi].punits, q4 = s_p.mat[mi].q4;
    const unsigned row_bytes = (unsigned)s_p.mat[mi].row_bytes, ring = (unsigned)s_p.n_slots, back = (unsigned)s_p.window * ST_COPY, slot = (unsigned)s_p.slot_bytes;
    const uint8_t * src = W + (size_t)(mi == ST_GATHER ? 0 : s_first[mi]) * row_bytes;
    const int * rows = sh_rows();
    const bool gather = mi == ST_GATHER;
    unsigned k = cp.k, s = cp.s, par = cp.par, bs = cp.bs, bpar = cp.bpar;
    bool ok = true;
#pragma unroll 1
    for (int i = (int)(k - kbase); i < nslots; i += ST_COPY) {
        if (k >= back) {
            if (!timed_bar(s_full + bs, bpar)) { ok = false; break; }
            bs += ST_COPY;
            if (bs >= ring) { bs -= ring; bpar ^= 1u; }
        }
        if (k >= ring && !timed_bar(s_empty + s, par ^ 1u)) { ok = false; break; }
        unsigned char * dst = smem + s * slot;
        uint64_t * bar = s_full + s;
        if (pieces > 1) {                                             // one piece of a row: Q4_0 nibbles, then their scales
            const int row = i / pieces, first = (i - row * pieces) * punits, nu = min(punits, units - first);
            const uint8_t * from = gather ? (GATED && (row & 1) ? W2 : src) + (size_t)rows[GATED ? row >> 1 : row] * row_bytes : src + (size_t)row * row_bytes;
            const unsigned nb = (unsigned)nu * 16u, ns = q4 ? (unsigned)nu * 2u : 0u;
            mbar_expect_tx(bar, nb + ns);
            bulk_g2s(dst, from + (size_t)first * 16, nb, bar);
            if (q4) bulk_g2s(dst + nb, from + (size_t)units * 16 + (size_t)first * 2, ns, bar);
        } else {
            const int n = min(rps, nrow - i * rps);
            mbar_expect_tx(bar, (unsigned)n * row_bytes);
            if (!gather) bulk_g2s(dst, src + (size_t)(i * rps) * row_bytes, (unsigned)n * row_bytes, bar);
            else {
#pragma unroll 1
                for (int r = 0; r < n; r++) {                         // up and gate rows in turn
                    const int v = i * rps + r;
                    bulk_g2s(dst + (unsigned)r * row_bytes, (GATED && (v & 1) ? W2 : src) + (size_t)rows[GATED ? v >> 1 : v] * row_bytes, row_bytes, bar);
                }
            }
        }
        k += ST_COPY;
        s += ST_COPY;
        if (s >= ring) { s -= ring; par ^= 1u; }
    }
    cp.k = k; cp.s = s; cp.par = par; cp.bs = bs; cp.bpar = bpar;
    return ok;
}

template <bool GATED>
__device__ __noinline__ void copy_weights(unsigned me) {
    const int second = s_p.falcon ? ST_FC1 : ST_WO, third = s_p.falcon ? ST_FC2 : ST_FC1, fourth = s_p.falcon ? ST_WO : ST_FC2;
    const int n = 5 * s_p.n_layer;
    Copier cp = {me, me, 0u, me, 0u};
    unsigned kbase = 0;
    bool ok = true;
#pragma unroll 1
    for (int i = 0, l = 0, m = 0; i <= n && ok; i++) {
        const StepLayer & L = s_p.layers[min(l, s_p.n_layer - 1)];
        const int mi = i == n ? ST_HEAD : (m == 0 ? ST_QKV : (m == 1 ? second : (m == 2 ? third : (m == 3 ? fourth : ST_GATHER))));
        const uint8_t * W = i == n ? s_p.head : L.w[m == 4 ? ST_UP : mi], * W2 = L.w[ST_GATE];
        if (m == 4 && !timed_bar(&s_listed, (unsigned)l & 1u)) { ok = false; break; }
        int nrow = s_rows[mi], nslots = s_slots[mi];
        if (m == 4) { const unsigned g = s_gather; nrow = (int)(g & 0xffffu); nslots = (int)(g >> 16); }   // (one word: see the head of the file)
        ok = issue<GATED>(mi, W, W2, kbase, nrow, nslots, cp);
        kbase += (unsigned)nslots;
        if (m == 4 && ok) mbar_arrive(&s_taken);
        if (++m == 5) { m = 0; l++; }
    }
    // (also when a wait ran out, here or elsewhere) do not leave with copies still on their way: this copier's slots that nobody fills again
    const unsigned ring = (unsigned)s_p.n_slots, end = ok ? kbase : cp.k - ST_COPY + 1u;
#pragma unroll 1
    for (unsigned j = cp.k; j >= ST_COPY && end - (j - ST_COPY) <= ring; j -= ST_COPY) {
        int spins = 0;
        while (!mbar_try_wait(s_full + (j - ST_COPY) % ring, ((j - ST_COPY) / ring) & 1u) && ++spins < (1 << 16)) {}
    }
    if (ok && me == 0) timed_bar(&s_done, 0u);                        // the clock runs to the end
}

// ------------------------------------------------------------------------------------------------ the kernel

template <int WT, bool GATED>
__global__ void __launch_bounds__(ST_THREADS, 1) k_step(const __grid_constant__ StepP args) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    static_assert(sizeof(StepP) % 8 == 0 && sizeof(StepP) / 8 <= ST_THREADS, "copied in one go");
    if (tid < (int)(sizeof(StepP) / 8)) reinterpret_cast<u64 *>(&s_p)[tid] = reinterpret_cast<const u64 *>(&args)[tid];
    if (tid < (int)(sizeof(StepLayer) / 8)) reinterpret_cast<u64 *>(&s_layer[0])[tid] = reinterpret_cast<const u64 *>(args.layers)[tid];
    if (tid < ST_GATHER) {                                            // rows [r0, r1) of every dense matrix
        const StepMat & m = args.mat[tid];
        const int g = (m.rows + m.gran - 1) / m.gran;
        const int r0 = min(m.rows, (int)(blockIdx.x * (unsigned)g / gridDim.x) * m.gran), r1 = min(m.rows, (int)((blockIdx.x + 1) * (unsigned)g / gridDim.x) * m.gran);
        s_first[tid] = r0; s_rows[tid] = r1 - r0;
        s_slots[tid] = mat_slots(m, r1 - r0);
    }
    if (tid == 0) {
        s_dead = 0; s_gather = 0u;
        const unsigned c8n = (unsigned)args.d / 8u;
        s_col0 = (int)(blockIdx.x * c8n / gridDim.x) * 8;
        s_ncol = (int)((blockIdx.x + 1) * c8n / gridDim.x) * 8 - s_col0;
        s_step = *args.step_no;                                       // raised by the CTA that finishes the step last
        atomicAdd(args.arrived, 1u);
        for (int s = 0; s < args.n_slots; s++) { mbar_init(s_full + s, 1); mbar_init(s_empty + s, ST_WARPS); }
        mbar_init(&s_listed, 1); mbar_init(&s_taken, ST_COPY); mbar_init(&s_done, ST_WARPS);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    if (wid >= ST_WARPS) {
        if (lane == 0) copy_weights<GATED>((unsigned)(wid - ST_WARPS));
        return;
    }
    // ================================================================= the computing warps
    const unsigned ep0 = s_step * (unsigned)(s_p.n_layer + 1) + 1u;   // number of the step's first layer
    int token, pos;
    if (s_p.fed) {
        token = s_p.token; pos = s_p.pos;
        if (blockIdx.x == 0 && tid == 0) { *s_p.tokens = token; *s_p.positions = pos; }
    } else { token = *s_p.tokens; pos = *s_p.positions; }
    embed_phase(token, pos, ep0);
    unsigned kbase = 0;
#pragma unroll 1
    for (int l = 0; l < s_p.n_layer; l++) {
        const StepLayer & L = s_layer[l & 1];
        const unsigned tag = ep0 + (unsigned)l;
        const u64 * x_in = s_p.x + (size_t)(l & 1) * s_p.d;
        {   // ---- vectors this layer reads once: into L2, spread over the CTAs (they are cold, and every CTA will want them)
            const int i = blockIdx.x * ST_CT + tid, lines = s_p.d / 32;
            const float * f = i < lines * 4 ? L.f[i / lines] : nullptr;
            if (f) asm volatile("prefetch.global.L2 [%0];" :: "l"(f + (size_t)(i % lines) * 32));
        }
        auto attention = [&]() {
#pragma unroll 1
            for (int h = blockIdx.x; h < s_p.n_head; h += gridDim.x) {
                if (s_p.hd == 128) attention_head<4>(h, l, pos, 0, tag);
                else               attention_head<2>(h, l, pos, 0, tag);
            }
        };
        // ---- the norm that opens the layer; QKV
        if (s_p.falcon) {                                             // attn_norm feeds the FFN, attn_norm2 (or it) the attention; the predictor reads x (llama.cpp:5422-5428)
            norm_any(x_in, tag, {L.f[ST_N1W], L.f[ST_N1B], smem + s_p.off_a, L.f[ST_N2W], L.f[ST_N2B], L.f[ST_N2W] ? smem + s_p.off_c : nullptr, smem + s_p.off_b, WT});
        } else {
            norm_any(x_in, tag, {L.f[ST_N1W], L.f[ST_N1B], smem + s_p.off_c, nullptr, nullptr, nullptr, nullptr, WT});
        }
        qkv_phase<WT>(l, kbase, tag);
        kbase += s_slots[ST_QKV];
        if (l + 1 < s_p.n_layer && wid == ST_WARPS - 1 && lane < (int)(sizeof(StepLayer) / 8))
            reinterpret_cast<u64 *>(&s_layer[(l + 1) & 1])[lane] = reinterpret_cast<const u64 *>(s_p.layers + l + 1)[lane];
        if (s_p.falcon) {
            // the two branches do not depend on each other: the predictor's first product before the attention, which hides its hand-over
            fc1_phase(l, kbase, tag);
            kbase += s_slots[ST_FC1];
            attention();
            fc2_phase(l, kbase, tag);
            kbase += s_slots[ST_FC2];
            wo_phase<WT>(l, kbase, tag);
            kbase += s_slots[ST_WO];
        } else {
            attention();
            wo_phase<WT>(l, kbase, tag);
            kbase += s_slots[ST_WO];
            // ---- ffn_inp = attention + x: its norm, and ffn_inp itself for the predictor
            norm_any(s_p.x2 + (size_t)(l & 1) * s_p.d, tag, {L.f[ST_N2W], L.f[ST_N2B], smem + s_p.off_a, nullptr, nullptr, nullptr, smem + s_p.off_b, WT});
            fc1_phase(l, kbase, tag);
            kbase += s_slots[ST_FC1];
            fc2_phase(l, kbase, tag);
            kbase += s_slots[ST_FC2];
        }
        // ---- the sparse FFN
        const int n = scan_words(s_p.maskw + (size_t)(l & 1) * (s_p.F / 8), tag);
        if (s_p.rows_total && blockIdx.x == 0 && tid == 0 && n) atomicAdd(s_p.rows_total, (u64)n);
        gather_list<GATED>(l, n);
        gather_phase<WT, GATED>(l, kbase, tag);
        kbase += s_slots[ST_GATHER];
        axpy_phase<WT>(l, n, tag);
        reduce_phase(l, tag);
    }
    // ---- output norm, lm head, greedy choice
    norm_any(s_p.x + (size_t)(s_p.n_layer & 1) * s_p.d, ep0 + (unsigned)s_p.n_layer, {s_p.out_w, s_p.out_b, smem + s_p.off_a, nullptr, nullptr, nullptr, nullptr, s_p.head_type});
    head_phase<WT>(kbase);
}

// ------------------------------------------------------------------------------------------------ plan and launch

static_assert(ST_SLICE == SLICE && QK == 32, "the plan counts in the kernels' slices and blocks");

StepDevice step_device() {
    StepDevice r = {0, 0, 80};
    int dev = 0, most = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) { cudaGetLastError(); return r; }
    r.sms = sm_count(); r.smem = (size_t)most;
    if (const char * v = getenv("PI_STEP_WINDOW")) r.window_kb = atoi(v);
    return r;
}

typedef void (*StepKernel)(const StepP);
static StepKernel step_kernel(bool q4, bool gated) {
    if (q4) return gated ? k_step<PI_TYPE_Q4_0, true> : k_step<PI_TYPE_Q4_0, false>;
    return gated ? k_step<PI_TYPE_F16, true> : k_step<PI_TYPE_F16, false>;
}

// A context or a stream can have a part of the device only (a green context).  No answer counts as the whole.
template <typename F> static F driver_call(const char * name) {
    void * f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion(name, &f, 12040, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) { cudaGetLastError(); return nullptr; }
    return (F)f;
}
static int context_sms() {
    static const auto current = driver_call<CUresult (*)(CUcontext *)>("cuCtxGetCurrent");
    static const auto resource = driver_call<CUresult (*)(CUcontext, CUdevResource *, CUdevResourceType)>("cuCtxGetDevResource");
    CUcontext ctx = nullptr;
    CUdevResource r;
    if (!current || !resource || current(&ctx) != CUDA_SUCCESS || !ctx || resource(ctx, &r, CU_DEV_RESOURCE_TYPE_SM) != CUDA_SUCCESS) return sm_count();
    return (int)r.sm.smCount;
}
static bool stream_has_sms(cudaStream_t st, int need) {
    static const auto green = driver_call<CUresult (*)(CUstream, CUgreenCtx *)>("cuStreamGetGreenCtx");
    static const auto resource = driver_call<CUresult (*)(CUgreenCtx, CUdevResource *, CUdevResourceType)>("cuGreenCtxGetDevResource");
    CUgreenCtx g = nullptr;
    CUdevResource r;
    if (!st || !green || !resource || green(st, &g) != CUDA_SUCCESS || !g || resource(g, &r, CU_DEV_RESOURCE_TYPE_SM) != CUDA_SUCCESS) return true;
    return (int)r.sm.smCount >= need;
}

bool step_fits(const StepPlan & pl, bool q4, bool gated) {
    const StepKernel kern = step_kernel(q4, gated);
    int dev = 0, cooperative = 0, per_sm = 0;
    cudaFuncAttributes at;
    const bool ok = cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && cooperative &&
                    cudaFuncGetAttributes(&at, kern) == cudaSuccess && at.sharedSizeBytes <= (size_t)ST_STATIC &&
                    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(step_device().smem - ST_STATIC)) == cudaSuccess &&
                    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, ST_THREADS, pl.smem) == cudaSuccess;
    if (!ok) cudaGetLastError();
    return ok && per_sm * context_sms() >= pl.grid;
}

int launch_step(const StepP & p, const StepPlan & pl, bool gated, cudaStream_t st) {
    if (!stream_has_sms(st, pl.grid)) return STEP_REFUSED;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pl.grid); cfg.blockDim = dim3(ST_THREADS); cfg.dynamicSmemBytes = pl.smem; cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;                      // the CTAs wait for one another: all are resident, or the launch fails
    attr[0].val.cooperative = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, step_kernel(p.q4, gated), p);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources || e == cudaErrorNotSupported) { cudaGetLastError(); return STEP_REFUSED; }
    PI_CUDA(e);
    return PI_OK;
}

}  // namespace pi
