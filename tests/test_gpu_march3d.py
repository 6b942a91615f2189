"""Route of the FP64 3-D step: grids that march along z (30 x 10 column blocks,
runs of planes), at the blocks' edges and one cell less and more, against the
oracle; and grids of few tiles, which stay on the tile kernel."""
import numpy as np
import pytest

from cases import rel_l1
from heraclespp_b200 import Domain
from oracle import Oracle
from test_gpu_march64 import BC3, PHYS, flow
from test_gpu_still_gas import us_per_step

pytestmark = pytest.mark.gpu

# more waves of tiles than the march needs plane steps for: full and partial
# blocks, a last run of one plane
MARCH = [([30, 10, 200], 0), ([29, 9, 200], 1), ([119, 29, 20], 0), ([151, 59, 10], 1), ([59, 39, 61], 0), ([61, 41, 61], 1)]


@pytest.mark.parametrize("lim,rs", PHYS)
@pytest.mark.parametrize("nx,b", MARCH)
def test_march_matches_oracle(nx, b, lim, rs):
    kw = dict(gamma=1.4, limiter=lim, riemann=rs, bc=BC3[b], xmax=(1.0, 0.7, 1.3),
              g=(0.03, -0.05, 0.02) if b else (0.0, 0.0, 0.0))
    ng = 3 if b else 2
    o = Oracle(3, nx, ng=ng, **kw)
    rho, rhou, E, fx = o.init_from_prim(*flow(o, 5 + nx[0]))
    start = (rho.copy(), rhou.copy(), E.copy())
    _, it, st, dts = o.run(rho, rhou, E, fx, cfl=0.3, max_iter=3, record_dts=True)
    assert (it, st) == (3, 0)
    d = Domain(3, nx, nghost=ng, precision="fp64", **kw)
    d.set_state(*start)
    d.run(cfl=0.3, nsteps=3)
    assert np.array_equal(d.dt_log()[:3], dts)
    for a, ref in zip(d.get_state(), (rho, rhou, E)):
        assert np.array_equal(a, ref)
    d = Domain(3, nx, nghost=ng, precision="fp64_fast", **kw)
    d.set_state(*start)
    d.run(nsteps=3, dts=dts)
    for a, ref in zip(d.get_state(), (rho, rhou, E)):
        assert rel_l1(a, ref) < 1e-12  # the bound of the fast FP64 tests


@pytest.mark.parametrize("prec", ["fp64", "fp64_fast"])
def test_small_grids_stay_on_tiles(prec):
    """A step of 32^3 cells is one wave of tiles, of 48^3 cells three: a good third
    of the time (with half as much again for the fixed part and the spread), which
    a march of three planes per CTA cannot give."""
    us = []
    for n in (32, 48):
        d = Domain(3, [n] * 3, gamma=1.4, limiter="VanLeer", riemann="HLLC", bc=["Periodic"] * 6, precision=prec)
        us.append(us_per_step(d, flow(d, n), 60))
    assert us[0] < 0.6 * us[1]
