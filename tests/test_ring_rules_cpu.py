"""The GEMMs' shared-memory rings (csrc/ring_rules.h, compiled here with the host compiler): whoever waits for a slot knows that
the slot's previous fill has completed, whatever the order in which the copies in flight complete.  The walk of the groups of
weight warps through tiles, k-tiles and slots is the kernels', restated."""
import ctypes
import os
import shutil
import subprocess

import pytest

from autogptq.tvm_b200 import build

SHIM = """
#include "ring_rules.h"
using namespace b200gptq;
extern "C" {
void rings(int bits, int groups, int rows, int several_tiles, int* out) {
    const PairRings r = pair_rings(bits, groups, rows, several_tiles != 0);
    out[0] = r.acc_sets; out[1] = r.stages; out[2] = r.slots;
}
int whole_turns(int stages, int groups) { return ring_in_whole_turns(stages, groups); }
int turns(int k_tiles) { return pair_turns(k_tiles); }
}
"""
CXX = os.environ.get("CXX", "g++")
pytestmark = pytest.mark.skipif(shutil.which(CXX) is None, reason="needs the host compiler")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("rings")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run([CXX, "-std=c++17", "-shared", "-fPIC", "-I", build.CSRC, str(d / "shim.cpp"), "-o", str(d / "shim.so")], check=True)
    return ctypes.CDLL(str(d / "shim.so"))


def _blind(units, slots, stages, groups=4, tiles=None):
    """The first (group, unit of 128 rows, "slot" or "stage") that waits without knowing that the fill before has completed; None where
    there is none.  Groups of weight warps take units in turn, through one tile of `units` after the other; a wait for a slot shows that
    its fill has come, a wait for a stage that the products of `stages` units before have retired, and products retire in order."""
    for g in range(groups):
        turn, base, seen, upto = g, 0, set(), -1
        for _ in range(tiles or 200 // units + 2):
            while turn < units:
                u = base + turn
                if u >= slots and u - slots not in seen:
                    return g, u, "slot"
                if u >= 2 * stages and u - 2 * stages > upto:
                    return g, u, "stage"
                seen.add(u)
                upto = max(upto, u - stages)
                turn += groups
            turn, base = turn - units, base + units
    return None


def _pair_rings(lib):
    """(bits, groups in a slot, rows per tile, several tiles per pair of SMs) -> (sets of accumulators, k-tiles of stages, slots)."""
    r = (ctypes.c_int * 3)()
    for bits in (2, 3, 4, 8):
        for groups in (1, 2, 3, 4):
            for rows in range(32, 257, 32):
                for several in (0, 1):
                    lib.rings(bits, groups, rows, several, r)
                    yield (bits, groups, rows, several), tuple(r)


def test_pair_rings_never_wait_blind(lib):
    """(a tile with an odd number of k-tiles ends in a unit of one)"""
    for what, (_, stages, slots) in _pair_rings(lib):
        assert stages % 2 == 0
        for k_tiles in (1, 2, 3, 5, 64, 171):
            assert _blind(lib.turns(k_tiles) // 2, slots, stages // 2) is None, (what, k_tiles)


def test_the_walk_finds_other_rings_at_fault():
    """(the check itself: slots that are no multiple of the groups, or fewer stages than groups, are not safe)"""
    assert _blind(32, 8, 4) is None
    for slots in (5, 6, 10):
        assert _blind(32, slots, 4)[2] == "slot"
    assert _blind(1, 10, 4, tiles=40)[2] == "slot"
    assert _blind(32, 8, 3)[2] == "stage"


def test_every_pair_ring_fits(lib):
    for (bits, groups, rows, several), (sets, stages, slots) in _pair_rings(lib):
        assert sets == (2 if rows <= 128 and several else 1)
        assert sets * rows + 32 * stages <= 512 and slots in (4, 8, 12, 16) and 8 <= stages <= 14
        slot = 4 * bits * 512 + groups * 384
        assert stages * rows * 64 + slots * slot + 1024 <= 222 * 1024


def test_stages_of_the_small_gemm_belong_to_one_group_each(lib):
    for stages in range(4, 24):
        s = lib.whole_turns(stages, 3)
        assert 3 <= s <= stages and all((kt - s) % 3 == kt % 3 for kt in range(s, 200))
