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
void rings(int bits, int groups, int rows, int k_tiles, int* out) {
    const PairRings r = pair_rings(bits, groups, rows, k_tiles);
    out[0] = r.acc_sets; out[1] = r.stages; out[2] = r.slots; out[3] = r.ahead;
}
int whole_turns(int stages, int groups) { return ring_in_whole_turns(stages, groups); }
int slot_step(int k_tiles) { return pair_slot_step(k_tiles); }
int fill_ahead(int slots, int step) { return pair_fill_ahead(slots, step); }
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


def _walk(k_tiles, tiles, groups=4):
    """Per group of weight warps: the slots' units it waits for, in order, through `tiles` tiles of `k_tiles` k-tiles."""
    out = []
    for g in range(groups):
        kt, base, units = g, 0, []
        for _ in range(tiles):
            while kt < k_tiles:
                units.append(base + (kt >> 1))
                kt += groups
            kt -= k_tiles
            base += (k_tiles + 1) // 2
        out.append(units)
    return out


def _first_blind_wait(k_tiles, tiles, slots, ahead):
    """The first (group, unit) whose slot may still be waiting for its previous fill; None where there is none."""
    for g, units in enumerate(_walk(k_tiles, tiles)):
        seen, upto = set(), -1          # fills this group has seen complete; all up to `upto` it knows of
        for u in units:
            if u >= slots and u - slots > upto and u - slots not in seen:
                return g, u
            seen.add(u)
            upto = max(upto, u - ahead)
    return None


def test_pair_rings_never_wait_blind(lib):
    for k_tiles in list(range(1, 40)) + [64, 65, 171, 172]:
        tiles = max(3, 400 // k_tiles)
        step = lib.slot_step(k_tiles)
        walks = [b - a for u in _walk(k_tiles, tiles) for a, b in zip(u, u[1:])]
        assert max(walks) <= step
        for slots in range(4 if step == 2 else 5, 17):
            assert _first_blind_wait(k_tiles, tiles, slots, lib.fill_ahead(slots, step)) is None, (k_tiles, slots)


def test_the_walk_finds_an_unlimited_ring_at_fault():
    """(the check itself: with every slot in flight an odd number of slots, or an odd number of k-tiles, is not safe)"""
    assert _first_blind_wait(64, 4, 5, 5) is not None
    assert _first_blind_wait(1, 40, 11, 11) is not None
    assert _first_blind_wait(33, 8, 6, 6) is not None
    assert _first_blind_wait(64, 4, 6, 6) is None


def test_every_pair_ring_fits(lib):
    r = (ctypes.c_int * 4)()
    for bits in (2, 3, 4, 8):
        for groups in (1, 2, 3, 4):
            for rows in range(32, 257, 32):
                for k_tiles in (1, 2, 3, 64):
                    lib.rings(bits, groups, rows, k_tiles, r)
                    sets, stages, slots, ahead = r
                    assert sets * rows + 32 * stages <= 512 and 4 <= slots <= 16 and 4 <= stages <= 14 and ahead >= 1
                    assert _first_blind_wait(k_tiles, max(3, 160 // k_tiles), slots, ahead) is None
                    slot = 4 * bits * 512 + groups * 384
                    assert stages * rows * 64 + slots * slot + 1024 <= 222 * 1024


def test_stages_of_the_small_gemm_belong_to_one_group_each(lib):
    for stages in range(4, 24):
        s = lib.whole_turns(stages, 3)
        assert 3 <= s <= stages and all((kt - s) % 3 == kt % 3 for kt in range(s, 200))
