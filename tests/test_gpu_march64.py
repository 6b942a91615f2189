"""The FP64 march kernels (Cartesian 2-D and 3-D) against the oracle: sizes at
the edges of their tiles (28-column warps in 2-D, 30 x 10 column blocks in
3-D), one cell less and more, and the smallest grids (two cells)."""
import numpy as np
import pytest

from cases import rel_l1
from heraclespp_b200 import Domain, setups
from oracle import Oracle

pytestmark = pytest.mark.gpu

BC2 = [["Periodic"] * 4, ["NullGradient", "Reflexive", "Reflexive", "NullGradient"]]
BC3 = [["Periodic"] * 6, ["NullGradient", "Reflexive", "Reflexive", "NullGradient", "Reflexive", "NullGradient"]]
G2D = [([2, 2], 0), ([27, 5], 1), ([28, 3], 0), ([29, 34], 1), ([57, 41], 1)]
G3D = [([2, 2, 2], 0), ([29, 9, 3], 1), ([30, 10, 7], 0), ([31, 11, 12], 1), ([33, 21, 5], 1)]
PHYS = [("VanLeer", "HLLC"), ("Minmod", "HLL"), ("VanAlbada", "Low Mach"), ("Constant", "HLLC")]


def flow(o, seed):
    """Smooth flow with a resting, uniform corner (zero differences and zero
    velocities) and jumps."""
    rng = np.random.default_rng(seed)
    rho, u, P = setups.Grid.from_domain(o).alloc()
    rho[...] = 1 + 0.3 * rng.uniform(-1, 1, rho.shape)
    P[...] = 1 + 0.3 * rng.uniform(-1, 1, rho.shape)
    for d in range(o.ndim):
        u[d] = 0.8 * rng.uniform(-1, 1, rho.shape)
    n = rho.shape
    corner = tuple(slice(0, (m + 1) // 2) for m in n)
    rho[corner], P[corner] = 1.0, 1.0
    u[(slice(None),) + corner] = 0.0
    return rho, u, P


@pytest.mark.parametrize("lim,rs", PHYS)
@pytest.mark.parametrize("nx,b", G2D + G3D)
def test_march_matches_oracle(nx, b, lim, rs):
    nd = len(nx)
    kw = dict(gamma=1.4, limiter=lim, riemann=rs, bc=(BC2 if nd == 2 else BC3)[b], xmax=(1.0, 0.7, 1.3),
              g=(0.03, -0.05, 0.02) if b else (0.0, 0.0, 0.0))
    o = Oracle(nd, nx, **kw)
    prim = flow(o, 5 + nx[0])
    rho, rhou, E, fx = o.init_from_prim(*prim)
    start = (rho.copy(), rhou.copy(), E.copy())
    _, it, st, dts = o.run(rho, rhou, E, fx, cfl=0.3, max_iter=6, record_dts=True)
    assert (it, st) == (6, 0)
    d = Domain(nd, nx, precision="fp64", **kw)
    d.set_state(*start)
    d.run(cfl=0.3, nsteps=6)
    got = d.get_state()
    assert np.array_equal(d.dt_log()[:6], dts)
    for a, ref in zip(got, (rho, rhou, E)):
        assert np.array_equal(a, ref)
    # the fast forms round differently in each of ~1e3 operations per cell and
    # step: 1e-12, the bound of the fast FP64 tests
    d = Domain(nd, nx, precision="fp64_fast", **kw)
    d.set_state(*start)
    d.run(nsteps=6, dts=dts)
    for a, ref in zip(d.get_state(), (rho, rhou, E)):
        assert rel_l1(a, ref) < 1e-12
