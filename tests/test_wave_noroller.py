"""The rows pass without the roller has its own forms of the box-fed kernel (FP32:
four cells per thread and four rows per warp; FP64: two).  Equal to the
thread-copied kernel bit for bit over whole steps, on grids whose last block is
partial in x (4, 4 and 28 columns) and in y, with fewer bins than tile buffers,
than the planes of the theta window and than roller energies in flight; and a
ragged batch equal to its scenarios run alone."""
import copy

import numpy as np
import pytest

from xbeach_gpu_b200.abi import XBG_FP32, XBG_FP64, XBG_PHASE_WAVE
from xbeach_gpu_b200.model import Batch, Model
from xbeach_gpu_b200.scenarios import make_case, make_ensemble

pytestmark = pytest.mark.gpu

FIELDS = ["ee", "rr", "H", "E", "D", "DR", "R", "thetamean", "Fx", "Fy", "urms", "ust", "zs", "uu", "vv", "zb", "hh"]


def _setup(m, p, zb, bnd):
    m.set_wave_boundary(0, bnd["St"], bnd["q"], t0=0.0, tend=p.rtlength, Trep=bnd["Trep"])
    m.set_sealevel([0.0, 1e6], [0.0, 0.0], [0.0, 0.0])
    m.set_wind([0.0, 1e6], [0.0, 0.0], [0.0, 0.0])
    m.init_state(zb, 0.0, 0.0)


@pytest.mark.parametrize("precision", [XBG_FP32, XBG_FP64])
@pytest.mark.parametrize("nx,ny,nt", [(68, 37, 7), (100, 12, 2), (36, 9, 1), (60, 26, 12)])
def test_box_tiles_equal_thread_copied_tiles(nx, ny, nt, precision):
    p, zb, bnd = make_case("linear_beach", nx=nx, ny=ny, ntheta=nt)
    p.roller = 0
    runs = []
    for variant in (0, 1):
        m = Model(p, precision)
        _setup(m, p, zb, bnd)
        m.set_variant(XBG_PHASE_WAVE, variant)
        m.advance(40)
        t, dt, n, _, rc = m.time()
        assert rc == 0 and n == 40
        runs.append((t, dt, {f: m.get(f).copy() for f in FIELDS}))
        m.close()
    assert runs[0][:2] == runs[1][:2]
    for f in FIELDS:
        assert np.array_equal(runs[0][2][f], runs[1][2][f]), f


@pytest.mark.parametrize("precision", [XBG_FP32, XBG_FP64])
def test_ragged_batch(precision):
    sc = []
    for p, zb, bnd in make_ensemble(4, seed=7, nx_range=(64, 192), ny_range=(32, 96), ntheta=9, dtbc=5.0):
        p = copy.copy(p)
        p.roller = 0
        sc.append((p, zb, bnd))
    b = Batch([p for p, _, _ in sc], precision)
    for s, (p, zb, bnd) in enumerate(sc):
        _setup(b.scenario(s), p, zb, bnd)
    b.advance(40)
    assert not b.status()["status"].any()
    for s, (p, zb, bnd) in enumerate(sc):
        m = Model(p, precision)
        _setup(m, p, zb, bnd)
        m.advance(40)
        for f in FIELDS:
            assert np.array_equal(b.scenario(s).get(f), m.get(f)), (s, f)
        m.close()
    b.close()
