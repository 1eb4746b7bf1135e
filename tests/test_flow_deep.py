"""The flow correction pass skips the window minima in blocks that lie deeper than the
offshore level less a metre.  The same state with that level far above the water,
which leaves every block to the minima, gives the same bits: on grids with whole and
ragged tiles, smaller than a tile, and with a dry shore."""
import numpy as np
import pytest

from xbeach_gpu_b200.abi import XBG_FP32, XBG_FP64
from xbeach_gpu_b200.model import Model
from xbeach_gpu_b200.scenarios import make_case

pytestmark = pytest.mark.gpu

AFTER = ["zs", "uu", "vv", "hh", "hu", "hv", "qx", "qy", "dzsdt"]


@pytest.mark.parametrize("precision", [XBG_FP32, XBG_FP64])
@pytest.mark.parametrize("nx,ny", [(128, 48), (101, 37), (24, 6)])
def test_deep_blocks_equal_minima(nx, ny, precision):
    p, zb, bnd = make_case("linear_beach", nx=nx, ny=ny, ntheta=8)
    m = Model(p, precision)
    m.set_wave_boundary(0, bnd["St"], bnd["q"], t0=0.0, tend=p.rtlength, Trep=bnd["Trep"])
    m.set_sealevel([0.0, 1e6], [0.0, 0.0], [0.0, 0.0])
    m.set_wind([0.0, 1e6], [0.0, 0.0], [0.0, 0.0])
    m.init_state(zb, 0.0, 0.0)
    m.advance(60)
    start = m.save_state()
    out, edge = [], None
    for level in (0.0, 1000.0):
        m.load_state(start)
        m.set_sealevel([0.0, 1e6], [level, level], [level, level])
        m.compute_dt()
        m.wave_boundary()
        m.flow_boundary()
        if edge is None:
            edge = {f: m.get(f) for f in ("uu", "vv", "zs")}
        for f, v in edge.items():
            m.set(f, v)
        m.wave_step()
        m.flow_step()
        out.append({f: m.get(f) for f in AFTER})
    assert np.abs(out[0]["uu"]).max() > 0
    for f in AFTER:
        assert np.array_equal(out[0][f], out[1][f]), f
    m.close()
