"""A copy warp that leaves early waits for the last copy into every slot of its
ring: bulk copies complete in any order, so every copy whose slot was not used
again may still be under way.  The bookkeeping that the kernels' exits use, built
for the host, against a ring that is filled copy by copy: rings of the
convolution over rows (3 to 18 stages), of the tiled convolution and of the
weight gradient (3 to 24 slots), left at every point of the first rounds and
after long runs."""
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
    L.ring_parity.restype = C.c_uint
    return L


@pytest.mark.parametrize("slots", [3, 4, 5, 6, 8, 13, 18, 24])
def test_every_slot_waits_for_its_last_copy(ring, slots):
    rng = random.Random(slots)
    for n in list(range(4 * slots)) + [rng.randrange(100, 2000000) for _ in range(200)]:
        last = {q % slots: q for q in range(max(0, n - slots), n)}
        for slot in range(slots):
            q = ring.ring_last(n, slots, slot)
            assert q == last.get(slot, -1), (slots, n, slot)
            if q >= 0:
                assert ring.ring_parity(q, slots) == q // slots % 2
