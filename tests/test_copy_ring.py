"""A copy warp that leaves early waits for the last copy into every slot of its
ring: bulk copies complete in any order, so every copy whose slot was not used
again may still be under way.  The bookkeeping that the kernels' exits use, built
for the host, against a ring that is filled copy by copy: rings of the
convolution over rows (3 to 18 stages, groups of 3 to 30 boxes, the last group
whole, empty or in part), of the tiled convolution and of the weight gradient
(one copy at a time, 3 to 24 slots)."""
import ctypes as C
import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def ring(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("ring") / "ring.so")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-shared", "-fPIC",
                        "-I", os.path.join(ROOT, "xbeach_gpu_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cxx", "copy_ring.cpp"), "-o", so], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = C.CDLL(so)
    L.ring_last.argtypes = [C.c_int, C.c_uint, C.c_int, C.c_int]
    L.ring_parity.restype = C.c_uint
    return L


def _check(ring, slots, group, rows, some):
    last, n = {}, rows * group
    for q in list(range(max(0, n - slots), n)) + [n + c for c in range(group) if some >> c & 1]:
        last[q % slots] = q
    for slot in range(slots):
        q = ring.ring_last(n, some, slots, slot)
        assert q == last.get(slot, -1), (slots, group, rows, bin(some), slot)
        if q >= 0:
            assert ring.ring_parity(q, slots) == q // slots % 2


@pytest.mark.parametrize("group,slots", [(3, 18), (3, 5), (9, 18), (9, 14), (6, 9), (12, 18), (1, 3), (1, 6), (1, 24)])
def test_every_slot_waits_for_its_last_copy(ring, group, slots):
    rng = random.Random(group * 100 + slots)
    for rows in list(range(9)) + [rng.randrange(10, 200000) for _ in range(20)]:
        for some in {0, 1, (1 << group) - 1, (1 << group) - 2, 1 << (group - 1), rng.randrange(1 << group)}:
            _check(ring, slots, group, rows, some)
