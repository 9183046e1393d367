"""The plan of the one-launch decode step (csrc/pi_step_plan.h) over every shape that it accepts, walked by a program without CUDA.

A row larger than a ring slot goes through the ring in pieces, and the last piece is the shortest.  A lane of the kernel takes the units u0,
u0 + 32 w, ... of its piece and looks only whether the LAST of them is there: all earlier ones have to lie inside every piece, or the lane
multiplies what an earlier round left in the slot.  The program restates the lanes and counts how often each unit of a row is taken (once,
by exactly one lane), and checks the ring's own conditions: slots that hold what is copied into them at 16-byte boundaries, teams that
divide the ring, sums that fit their place, regions that fit the shared memory."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

WALK = r"""
#include <stdio.h>
#include <set>
#include <tuple>
#include <vector>
#include "pi_step_plan.h"
using namespace pi;

static long plans, mats, refused;
static bool fail(const char * what, const StepShape & s, int i, const StepMat & m) {
    printf("%s: wtype %d d %ld F %ld rank %ld hd %d: matrix %d units %d pieces %d punits %d wpr %d upt %d rps %d\n", what, s.wtype, (long)s.d, (long)s.F,
           (long)s.rank, s.hd, i, m.units, m.pieces, m.punits, m.wpr, m.upt, m.rps);
    return false;
}

static std::set<std::tuple<int, int, int, int, int>> seen;
static bool lanes(const StepMat & m) {
    if (!seen.insert({m.units, m.pieces, m.punits, m.wpr, m.upt}).second) return true;
    mats++;
    std::vector<int> taken(m.units, 0);
    for (int pc = 0; pc < m.pieces; pc++) {
        const int first = pc * m.punits, nq = m.punits < m.units - first ? m.punits : m.units - first;
        for (int part = 0; part < m.wpr; part++)
            for (int lane = 0; lane < 32; lane++) {
                const int u0 = part * 32 + lane, step = m.wpr * 32;
                const bool last_ok = u0 + (m.upt - 1) * step < nq;
                for (int j = 0; j < m.upt; j++) {
                    if (j == m.upt - 1 && !last_ok) break;
                    if (u0 + j * step >= nq) return false;
                    taken[first + u0 + j * step]++;
                }
            }
    }
    for (int u : taken) if (u != 1) return false;
    return true;
}

static bool check(const StepShape & s, const StepDevice & dev) {
    StepPlan p;
    if (!step_plan(s, dev, p)) { refused++; return true; }
    plans++;
    const int unit[ST_N_MAT] = {0, 0, 16, 16, 0, 0};
    for (int i = 0; i < ST_N_MAT; i++) {
        const StepMat & m = p.mat[i];
        const int ub = unit[i] ? unit[i] : (m.q4 ? 18 : 16), teams = ST_WARPS / m.wpr;
        if (!lanes(m)) return fail("a lane beyond its piece", s, i, m);
        if (m.wpr * teams != ST_WARPS || p.n_slots % teams || teams % m.pieces) return fail("teams", s, i, m);
        if (m.upt < 1 || m.upt > 4 || (m.upt > 2 && m.rps > 2) || (m.rps != 1 && m.rps != 2 && m.rps != 4)) return fail("rows at a time", s, i, m);
        if (m.pieces > 1 ? m.punits * ub > p.slot_bytes || m.rps != 1 || m.punits % 8 || (m.units - (m.pieces - 1) * m.punits) % (m.q4 ? 8 : 1)
                         : m.rps * m.row_bytes > p.slot_bytes) return fail("slot", s, i, m);
        if (m.row_bytes % 16 || m.chunk < 1 || m.chunk % m.gran || m.chunk % m.rps || m.chunk * m.wpr * m.pieces > ST_PART) return fail("sums", s, i, m);
    }
    const StepMat & qkv = p.mat[ST_QKV];                              // rows in pieces fill the slot but for a share of the last one
    if (qkv.pieces > 1 && (qkv.q4 || qkv.punits * 16 + 127 < p.slot_bytes)) return fail("pieces smaller than a slot", s, ST_QKV, qkv);
    if (p.n_slots > ST_MAX_SLOTS || p.n_slots % ST_COPY || p.window < 1 || p.window * ST_COPY > p.n_slots || p.slot_bytes % 128) return fail("ring", s, 0, p.mat[0]);
    if (p.smem + ST_STATIC > dev.smem || p.off_part + ST_PART * 4 > p.off_rows || p.off_rows + (int)((s.F + p.grid - 1) / p.grid) * 4 > (int)p.smem || p.off_a < p.n_slots * p.slot_bytes) return fail("shared memory", s, 0, p.mat[0]);
    if (p.grid > dev.sms || p.grid * 8 > s.d || p.grid * 8 > s.F || p.groups < 1 || p.wpt * ST_CT * 32 < s.F) return fail("grid", s, 0, p.mat[0]);
    return true;
}

int main() {
    const StepDevice dev = {148, 232448, 80};
    bool ok = true;
    for (int q4 = 0; q4 < 2; q4++)
        for (int64_t d = 512; d <= 16640; d += q4 ? 256 : 32)
            for (int64_t rank = 8; rank <= 8192; rank += 8)
                for (int hd = 64; hd <= 128; hd *= 2) {
                    if (d % hd) continue;
                    for (int falcon = 0; falcon < 2; falcon++) {
                        StepShape s = {q4 ? PI_TYPE_Q4_0 : PI_TYPE_F16, q4 && !falcon ? PI_TYPE_Q4_0 : PI_TYPE_F16, falcon, d, (d * 7 / 2 + 31) / 32 * 32, d, rank, 32000, hd, 2048};
                        ok = check(s, dev) && ok;
                    }
                }
    // few and many neurons, outputs and positions
    for (int q4 = 0; q4 < 2; q4++)
        for (int64_t d : {768, 1024, 2560, 4096, 5120, 7168, 8192, 9216, 12288})
            for (int64_t F : {32, 64, 992, 1024, 4128, 16384, 16416, 32768, 32800, 65536, 65568})
                for (int64_t vocab : {1, 7, 147, 149, 50272, 256000})
                    for (int n_ctx : {1, 63, 512, 2047, 3584, 3585}) {
                        StepShape s = {q4 ? PI_TYPE_Q4_0 : PI_TYPE_F16, q4 ? PI_TYPE_Q4_0 : PI_TYPE_F16, 0, d, F, d / 8, 1024, vocab, 128, n_ctx};
                        ok = check(s, dev) && ok;
                    }
    printf("%ld plans, %ld refused, %ld kinds of matrix\n", plans, refused, mats);
    return ok && plans > 100000 ? 0 : 1;
}
"""


def test_every_plan_takes_every_unit_of_a_row_once(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "walk.cpp", tmp_path / "walk"
    src.write_text(WALK)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-I", os.path.join(ROOT, "powerinfer_b200", "csrc"), str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout[-3000:]
