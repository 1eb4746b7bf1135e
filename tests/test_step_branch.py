"""The step graph runs a boundary kernel as a branch beside the dispersion pass: the
flow boundary, or without the flow the wave boundary.  A profiled step runs every
kernel in order, so the two must give the same state bit for bit, for one domain
and for a batch, and with the rows pass by box copies and by thread copies."""
import numpy as np
import pytest

from xbeach_gpu_b200.abi import XBG_FP32
from xbeach_gpu_b200.model import Batch, Model
from xbeach_gpu_b200.scenarios import make_case

pytestmark = pytest.mark.gpu

FIELDS = ["ee", "rr", "H", "D", "thetamean", "Fx", "Fy", "zs", "uu", "vv", "hh"]


@pytest.mark.parametrize("nx", [64, 45])
@pytest.mark.parametrize("flow", [0, 1])
def test_graph_equals_kernels_in_order(nx, flow):
    p, zb, bnd = make_case("linear_beach", nx=nx, ny=32, ntheta=5)
    p.flow, p.sedtrans = flow, 0

    def setup(m):
        m.set_wave_boundary(0, bnd["St"], bnd["q"], t0=0.0, tend=p.rtlength, Trep=bnd["Trep"])
        m.set_sealevel([0.0, 1e6], [0.0, 0.3], [0.0, 0.0])
        m.set_wind([0.0, 1e6], [0.0, 2.0], [0.0, 0.0])
        m.init_state(zb, 0.0, 0.0)
    runs = []
    for graph in (True, False):
        m, b = Model(p), Batch([p, p], XBG_FP32)
        setup(m)
        for s in (0, 1):
            setup(b.scenario(s))
        if graph:
            m.advance(30)
            b.advance(30)
        else:
            for _ in range(30):
                m.profile_step()
                b.profile_step()
        assert m.time()[2] == 30 and m.time()[4] == 0 and not b.status()["status"].any()
        runs.append([{f: h.get(f).copy() for f in FIELDS} for h in (m, b.scenario(0), b.scenario(1))])
        b.close()
        m.close()
    assert float(np.abs(runs[0][0]["H"]).max()) > 0.0
    for a, c in zip(*runs):
        for f in FIELDS:
            assert np.array_equal(a[f], c[f]), f
