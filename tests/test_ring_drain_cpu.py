"""What a kernel waits for before it ends although one of its waits ran out (csrc/pi_ring.h, ring_land): the copies of the last use of every ring
slot, and nothing else.  A program without CUDA walks rings of every size with a model of a barrier: a wait for a parity is over when the
current phase has the other one, so that a fresh barrier is "over" for parity 1."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "powerinfer_b200", "csrc")

WALK = r"""
#include <stdio.h>
#include "pi_ring.h"
static bool over(int completed, int parity) { return (completed & 1) != parity; }      // mbarrier.try_wait.parity after `completed` phases
int main() {
    for (int slots = 1; slots <= 16; slots++)
        for (int issued = 0; issued <= 5 * slots + 1; issued++)
            for (int slot = 0; slot < slots; slot++) {
                int uses = 0;
                for (int st = 0; st < issued; st++) uses += st % slots == slot;
                const int parity = pi::ring_last_parity(issued, slots, slot);
                if (uses == 0) { if (parity >= 0) { printf("%d %d %d: no use\n", slots, issued, slot); return 1; } continue; }
                // a slot is used again only when its former use is over: either all uses are, or all but the last
                if (parity < 0 || over(uses - 1, parity) || !over(uses, parity)) { printf("%d %d %d: parity %d of %d uses\n", slots, issued, slot, parity, uses); return 1; }
            }
    return 0;
}
"""


def test_the_last_use_of_every_slot_is_waited_for(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "walk.cpp", tmp_path / "walk"
    src.write_text(WALK)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-I", CSRC, str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout[-3000:]


def test_no_kernel_waits_for_either_parity():
    """`while (!try_wait(bar, 0) && !try_wait(bar, 1))` ends at once: one of the two is always over."""
    for name in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, name)).read()
        assert not re.search(r"try_wait\([^;]*, 0u?\) *&& *!mbar_try_wait\([^;]*, 1u?\)", text), name


def test_tensor_memory_is_given_back_when_no_product_is_in_flight():
    """Every kernel that gives tensor memory back lets the issuing warp wait for its last products, also after a wait ran out (no look at s_dead)."""
    seen = 0
    for name in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, name)).read()
        if "tc_dealloc(tmem" not in text:
            continue
        seen += 1
        assert re.search(r"tc_commit\(&(\w+)\);[^\n]*\n *for \(int spins = 0; spins < \(1 << 20\) && !mbar_try_wait\(&\1, 0u\); spins\+\+\) \{\}\n *__syncwarp\(\);", text), name
    assert seen == 3
