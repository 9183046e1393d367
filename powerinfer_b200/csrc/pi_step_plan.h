// The plan of the one-launch decode step (pi_step.cu): how a model's matrices go through the shared-memory ring.  Plain C++, so that a
// program without CUDA can walk it over every shape.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/powerinfer_b200.h"

namespace pi {

static constexpr int ST_QKV = 0, ST_WO = 1, ST_FC1 = 2, ST_FC2 = 3, ST_HEAD = 4, ST_GATHER = 5, ST_N_MAT = 6;   // what goes through the ring: dense matrices, the rows of the gather
static constexpr int ST_WARPS = 16, ST_CT = ST_WARPS * 32;          // computing warps / threads
static constexpr int ST_COPY = 4;                                     // copying warps: one lane gets through a slot in about 500 clocks
static constexpr int ST_THREADS = ST_CT + ST_COPY * 32;
static constexpr int ST_MAX_SLOTS = 48;
static constexpr int ST_PART = 2048;                                // floats of s_part
static constexpr int ST_LIST = 512;                                 // rows of a group that an axpy pass takes at once
static constexpr int ST_SLICE = 1024;                               // columns of an axpy slice: 32 sums per lane
static constexpr int ST_RED = 8 * 32 * 33 * 4;                      // bytes of the warps' column sums
static constexpr int ST_STATIC = 3072;                              // room for the kernel's static shared memory
static constexpr int ST_MIN_D = 768;                                  // narrower models: a layer's hand-overs cost as much as its launches (5 layers of d 512: 219
                                                                      // us against 195 by kernels, 3 layers of d 768: 150 against 157)

// a matrix cut for the ring: rows in units of `gran` dealt evenly to the CTAs; a slot holds `rps` rows (1, 2 or 4), or one of `pieces` pieces of
// a row (`punits` units; a unit is 8 columns of F16, a block of Q4_0) and is the work of a team of `wpr` warps, whose lanes take `upt` units
// each; `chunk` rows have room for their sums
struct StepMat { int rows, gran, units, rps, pieces, punits, wpr, upt, chunk, q4; int64_t row_bytes; };

struct StepShape { int wtype, head_type, falcon; int64_t d, F, dkv, rank, n_vocab; int hd, n_ctx; };
struct StepDevice { int sms; size_t smem; int window_kb; };          // shared memory that a block may ask for; KB on their way per SM
struct StepPlan {
    bool ok = false;
    StepMat mat[ST_N_MAT];
    int slot_bytes = 0, n_slots = 0, window = 0, grid = 0, groups = 0, wpt = 0;
    int off_a = 0, off_b = 0, off_c = 0, off_h = 0, off_part = 0, off_rows = 0;
    size_t smem = 0, words = 0;                                      // shared memory; bytes of the words passed between CTAs
};

inline int64_t step_row_bytes(int wtype, int64_t cols) { return wtype == PI_TYPE_Q4_0 ? cols / 32 * 18 : cols * 2; }

// How a matrix goes through a ring of n slots of `slot` bytes; wpr == 0: not at all.  A row is cut where it is larger than a slot; a team has as
// few warps as hold the activation in registers (4 units a lane), so that a warp's wait and sum come once per 2-4 KB.  A slot of the ring
// goes to the same team round by round, which has then seen the slot's round before itself.
inline StepMat step_mat_plan(int wtype, int64_t rows, int64_t cols, int gran, int slot, int n, int grid) {
    StepMat m{};
    m.q4 = wtype == PI_TYPE_Q4_0;
    m.rows = (int)rows; m.gran = gran; m.row_bytes = step_row_bytes(wtype, cols);
    m.units = m.q4 ? (int)(cols / 32) : (int)(cols / 8);
    const int unit_bytes = m.q4 ? 18 : 16;
    m.pieces = 1; m.punits = m.units;
    while ((int64_t)m.punits * unit_bytes > slot) {
        m.pieces *= 2;
        m.punits = ((m.units + m.pieces - 1) / m.pieces + 7) / 8 * 8;  // (a piece's scales are whole 16-byte words)
        if (m.pieces > ST_WARPS || m.punits * (m.pieces - 1) >= m.units) return m;
    }
    for (int w = 1; w <= ST_WARPS; w *= 2) {
        const int upt = (m.punits + 32 * w - 1) / (32 * w), teams = ST_WARPS / w;
        if (upt > 4 || n % teams || teams % m.pieces) continue;
        // a lane looks only for its last unit: the earlier ones have to lie inside every piece, the last and shortest one too
        if (m.units - (m.pieces - 1) * m.punits < (upt - 1) * 32 * w) continue;
        const int64_t per_cta = (rows + grid - 1) / grid;
        int64_t rps = m.pieces > 1 ? 1 : std::min<int64_t>(std::min<int64_t>(slot / m.row_bytes, upt <= 2 ? 4 : 2), std::max<int64_t>(1, (per_cta + teams - 1) / teams));
        if (rps == 3) rps = 2;
        if (rps > m.rps) { m.wpr = w; m.upt = upt; m.rps = (int)rps; }
    }
    if (!m.wpr) return m;
    int unit = m.rps;                                                 // whole slots, whole groups of `gran` rows
    while (unit % gran) unit += m.rps;
    m.chunk = ST_PART / (m.wpr * m.pieces) / unit * unit;
    return m;
}

inline size_t step_up128(size_t v) { return (v + 127) & ~size_t(127); }

// false: the shape is not eligible
inline bool step_plan(const StepShape & s, const StepDevice & dev, StepPlan & pl) {
    pl = StepPlan();
    if (dev.sms <= 0 || s.d < ST_MIN_D || s.d > 4 * ST_CT * 8 || s.F > 4 * 32 * ST_CT || s.F % 32 || s.n_ctx > 7 * ST_CT || (s.hd != 64 && s.hd != 128)) return false;
    const int grid = (int)std::min<int64_t>(dev.sms, std::min<int64_t>(s.F / 8, s.d / 8));
    if (grid < 1) return false;
    const bool q4 = s.wtype == PI_TYPE_Q4_0;
    if (s.d % (q4 ? 256 : 32) || s.rank % 8) return false;
    const size_t act = q4 ? (size_t)(s.d / 32) * 40 : (size_t)s.d * 2;
    const size_t act_head = s.head_type == PI_TYPE_Q4_0 ? (size_t)(s.d / 32) * 40 : (size_t)s.d * 2;
    const size_t a = step_up128(std::max(std::max(act, act_head), (size_t)ST_RED));
    const size_t att = (size_t)s.n_ctx * 6 + (size_t)ST_WARPS * s.hd * 4 + (size_t)3 * s.hd * 2 + ST_WARPS * 8 + 64;
    const int64_t myrow = (s.F + grid - 1) / grid + 1;
    const size_t lists = (size_t)(2 * (s.F / 32) + 1) * 4 + (size_t)4 * ST_LIST * 4 + 64, rows = step_up128((size_t)myrow * 4);
    const size_t b = step_up128(std::max(std::max((size_t)s.d * 2, att), lists));
    const size_t c = s.falcon ? step_up128(act) : 0;                  // else the first region serves: it is free until the FFN's norm
    const size_t h = step_up128((size_t)s.rank * 2), part = step_up128((size_t)ST_PART * 4);
    const size_t fixed = a + b + c + h + part + rows, room = dev.smem > ST_STATIC ? dev.smem - ST_STATIC : 0;
    if (fixed >= room) return false;
    // Slots of about 8 KB (F16) or 4.6 KB (Q4_0): smaller ones cost the copying warps more than they save, larger ones leave teams without
    // work at the end of a matrix (steps of the 7B, 40B and 70B shapes in 4, 8, 16 and 36 KB slots: 1030, 729, 785, 856; 724, 574, 807, 591;
    // 622, 639, 690, 736 us).  A row that is larger goes whole or in even pieces that fill the slot: what a slot does not hold is missing in
    // the ring, and a piece of half a slot costs the copying warps as much as a whole one.  Layers in 8 KB slots, in slots that the pieces fill,
    // by the launch sequence: F16, 3 of d 4352 265, 235, 261 us; 3 of d 5120 295, 265, 330; 3 of d 6656 357, 336, 417; 1 of d 9216 305, 242, 265;
    // 1 of d 10240 327, 272, 376 (12 KB slots: 3 of d 5632 311, in pieces of 5.5 KB 291).  Q4_0, in 6.9 KB slots, whole rows, by the
    // sequence: d 12544 341, 181, 198; d 13312 361, 186, 209.
    const int64_t row = step_row_bytes(s.wtype, s.d), units = s.d / (q4 ? 32 : 8), unit_bytes = q4 ? 18 : 16;
    if (q4 && row > 7680) return false;                               // (1 layer of d 14336, F 39936: 244 us in two pieces, 199 by the sequence)
    int64_t slot64 = q4 ? (row <= 4608 ? row * std::max<int64_t>(1, 4608 / row) : row) : 8192;
    if (!q4 && row > slot64) {
        int64_t pieces = 1;
        while (row > pieces * 10240) pieces *= 2;
        slot64 = ((units + pieces - 1) / pieces + 7) / 8 * 8 * unit_bytes;
    }
    const int slot = (int)((slot64 + 127) / 128 * 128);
    bool found = false;
    const int most_slots = (int)std::min<size_t>(ST_MAX_SLOTS, (room - fixed) / slot);
    for (int step = 16; step >= 4 && !found; step /= 2) {             // (teams of one, two, four warps)
        const int n = most_slots / step * step;
        if (n < 8 || 4 * n < 3 * most_slots) continue;
        const StepMat m[ST_N_MAT] = {
            step_mat_plan(s.wtype, s.d + 2 * s.dkv, s.d, 1, slot, n, grid), step_mat_plan(s.wtype, s.d, s.d, 1, slot, n, grid), step_mat_plan(PI_TYPE_F16, s.rank, s.d, 1, slot, n, grid),
            step_mat_plan(PI_TYPE_F16, s.F, s.rank, 8, slot, n, grid), step_mat_plan(s.head_type, s.n_vocab, s.d, 1, slot, n, grid), step_mat_plan(s.wtype, s.F, s.d, 2, slot, n, grid)};
        found = true;
        for (int i = 0; i < ST_N_MAT; i++) { found = found && m[i].wpr && m[i].chunk >= 1; pl.mat[i] = m[i]; }
        pl.slot_bytes = slot; pl.n_slots = n;
    }
    if (!found) return false;
    pl.window = std::max(1, std::min(pl.n_slots, dev.window_kb * 1024 / pl.slot_bytes) / ST_COPY);     // per copying warp
    pl.grid = grid;
    const int n_slices = (int)((s.d + ST_SLICE - 1) / ST_SLICE);
    pl.groups = std::min(64, grid / n_slices);
    if (pl.groups < 1) return false;
    const int64_t cols = ((s.d / 8 + grid - 1) / grid) * 8;
    if (cols > ST_CT || pl.groups * cols > ST_PART) return false;
    const size_t ring = step_up128((size_t)pl.n_slots * pl.slot_bytes);
    pl.off_a = (int)ring; pl.off_b = (int)(ring + a); pl.off_c = s.falcon ? (int)(ring + a + b) : pl.off_a;
    pl.off_h = (int)(ring + a + b + c); pl.off_part = (int)(ring + a + b + c + h); pl.off_rows = (int)(ring + a + b + c + h + part);
    pl.smem = ring + fixed;
    pl.wpt = s.F / 32 > 2 * ST_CT ? 4 : (s.F / 32 > ST_CT ? 2 : 1);
    // words: x, x2 [2][d] u64; qkv [2][d + 2 dkv] u64; h [2][F] u64; part [2][groups][d] u64; acto [2][d], acts [2][d / 32], hid [2][rank],
    // mask words [2][F / 8] u32
    pl.words = (size_t)2 * 8 * (s.d + s.d + s.d + 2 * s.dkv + s.F + (size_t)pl.groups * s.d) + (size_t)2 * 4 * (s.d + s.d / 32 + s.rank + s.F / 8) + 16 * 256;
    pl.ok = true;
    return true;
}

}  // namespace pi
