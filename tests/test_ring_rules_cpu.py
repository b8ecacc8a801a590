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
void rings(int bits, int groups, int rows, int* out) {
    const PairRings r = pair_rings(bits, groups, rows);
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


def _walk(k_tiles, tiles, turns, groups=4):
    """Per group of weight warps, turn by turn through `tiles` tiles of `k_tiles` k-tiles: the unit whose slot it waits for, and
    the k-tile's number among all (None: a turn without one).  `turns` per tile; the last slot of a tile may hold one k-tile."""
    out = []
    for g in range(groups):
        kt, units, real, steps, s = g, 0, 0, [], g
        for _ in range(tiles):
            while kt < turns:
                steps.append((units + (kt >> 1), real + kt if kt < k_tiles else None))
                assert steps[-1][1] is None or steps[-1][1] == s      # what the kernel counts its stages by
                kt, s = kt + groups, s + groups
            kt, s = kt - turns, s - (turns - k_tiles)
            units, real = units + (k_tiles + 1) // 2, real + k_tiles
        out.append(steps)
    return out


def _blind_slot(walk, slots):
    """The first (group, unit) that waits for a slot whose previous fill the group has not seen; None where there is none."""
    for g, steps in enumerate(walk):
        seen = set()
        for u, _ in steps:
            if u >= slots and u - slots not in seen:
                return g, u
            seen.add(u)
    return None


def _blind_stage(walk, stages):
    """The first (group, k-tile) that waits for the products of `stages` k-tiles before without knowing that those of twice as
    many before have retired.  Products retire in order, and a wait for k-tile r shows them up to r - stages."""
    for g, steps in enumerate(walk):
        upto = -1
        for _, r in steps:
            if r is None or r < stages:
                continue
            if r - 2 * stages > upto:
                return g, r
            upto = r - stages
    return None


def test_pair_rings_never_wait_blind(lib):
    for k_tiles in list(range(1, 40)) + [64, 65, 101, 171, 172]:
        walk = _walk(k_tiles, max(3, 400 // k_tiles), lib.turns(k_tiles))
        for slots in range(4, 17, 2):
            assert _blind_slot(walk, slots) is None, (k_tiles, slots)
        for stages in range(8, 15):
            assert _blind_stage(walk, stages) is None, (k_tiles, stages)
        # every slot is left by two turns, and every k-tile has one group
        units = [u for steps in walk for u, _ in steps]
        real = sorted(r for steps in walk for _, r in steps if r is not None)
        whole = [u for u in set(units) if u < max(units) - 2]
        assert all(units.count(u) == 2 for u in whole) and real == list(range(len(real)))


def test_the_walk_finds_other_rings_at_fault():
    """(the check itself: an odd number of slots, or tiles walked by their odd number of k-tiles, is not safe)"""
    assert _blind_slot(_walk(64, 4, 64), 5) is not None
    assert _blind_slot(_walk(64, 4, 64), 6) is None
    assert _blind_slot(_walk(33, 8, 33), 6) is not None
    assert _blind_slot(_walk(1, 40, 1), 10) is not None
    assert _blind_stage(_walk(64, 4, 64), 3) is not None


def test_every_pair_ring_fits(lib):
    r = (ctypes.c_int * 3)()
    for bits in (2, 3, 4, 8):
        for groups in (1, 2, 3, 4):
            for rows in range(32, 257, 32):
                lib.rings(bits, groups, rows, r)
                sets, stages, slots = r
                assert sets * rows + 32 * stages <= 512 and slots in range(4, 17, 2) and 8 <= stages <= 14
                slot = 4 * bits * 512 + groups * 384
                assert stages * rows * 64 + slots * slot + 1024 <= 222 * 1024


def test_stages_of_the_small_gemm_belong_to_one_group_each(lib):
    for stages in range(4, 24):
        s = lib.whole_turns(stages, 3)
        assert 3 <= s <= stages and all((kt - s) % 3 == kt % 3 for kt in range(s, 200))


def test_pair_units_never_wait_blind(lib):
    """Groups take whole units in turn, through one tile after the other (a tile with an odd number of k-tiles ends in a unit of one):
    a slot's previous fill was the group's own, and a stage's products of two rounds before have retired."""
    r = (ctypes.c_int * 3)()
    for bits in (2, 3, 4, 8):
        for groups in (1, 2, 3, 4):
            for rows in range(32, 257, 32):
                lib.rings(bits, groups, rows, r)
                stages, slots = r[1] // 2, r[2]
                assert r[1] % 2 == 0
                for k_tiles in (1, 2, 3, 5, 64, 171):
                    units = lib.turns(k_tiles) // 2
                    for g in range(4):
                        turn, base, seen, upto = g, 0, set(), -1
                        for _ in range(200 // units + 2):
                            while turn < units:
                                u = base + turn
                                assert u % 4 == g
                                assert u < slots or u - slots in seen
                                assert u < 2 * stages or u - 2 * stages <= upto
                                seen.add(u)
                                upto = u - stages
                                turn += 4
                            turn, base = turn - units, base + units
