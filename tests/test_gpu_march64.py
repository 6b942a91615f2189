"""The FP64 march kernels (1-D, Cartesian 2-D and 3-D) against the oracle: sizes
at the edges of their tiles (runs of 32 cells and more in 1-D, 28-column warps
in 2-D, 30 x 10 column blocks in 3-D), one cell less and more, and the smallest
grids (two cells)."""
import numpy as np
import pytest

from cases import rel_l1
from heraclespp_b200 import Domain, setups
from oracle import Oracle

pytestmark = pytest.mark.gpu

BC2 = [["Periodic"] * 4, ["NullGradient", "Reflexive", "Reflexive", "NullGradient"]]
BC3 = [["Periodic"] * 6, ["NullGradient", "Reflexive", "Reflexive", "NullGradient", "Reflexive", "NullGradient"]]
# 2-D grids march from more than 2 x 148 tiles of 16 x 16; the others run as tiles
G2D = [([2, 2], 0), ([29, 34], 1), ([251, 309], 1), ([252, 311], 0), ([253, 310], 1), ([3, 4800], 0), ([4760, 5], 1)]
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
    ng = 3 if b and min(nx) > 2 else 2
    o = Oracle(nd, nx, ng=ng, **kw)
    prim = flow(o, 5 + nx[0])
    rho, rhou, E, fx = o.init_from_prim(*prim)
    start = (rho.copy(), rhou.copy(), E.copy())
    _, it, st, dts = o.run(rho, rhou, E, fx, cfl=0.3, max_iter=6, record_dts=True)
    assert (it, st) == (6, 0)
    d = Domain(nd, nx, nghost=ng, precision="fp64", **kw)
    d.set_state(*start)
    d.run(cfl=0.3, nsteps=6)
    got = d.get_state()
    assert np.array_equal(d.dt_log()[:6], dts)
    for a, ref in zip(got, (rho, rhou, E)):
        assert np.array_equal(a, ref)
    # the fast forms round differently in each of ~1e3 operations per cell and
    # step: 1e-12, the bound of the fast FP64 tests
    d = Domain(nd, nx, nghost=ng, precision="fp64_fast", **kw)
    d.set_state(*start)
    d.run(nsteps=6, dts=dts)
    for a, ref in zip(d.get_state(), (rho, rhou, E)):
        assert rel_l1(a, ref) < 1e-12


@pytest.mark.parametrize("geom,bc,ng", [("Cartesian", ["Periodic"] * 2, 2), ("Cartesian", ["Reflexive", "NullGradient"], 3),
                                        ("Spherical", ["Reflexive", "NullGradient"], 2)])
@pytest.mark.parametrize("n", [3, 31, 32, 33, 65, 512, 513, 1000, 8192, 8193])
def test_1d_cluster_matches_oracle(n, geom, bc, ng):
    """Steps in one launch, across launches, to a time with outputs on the way,
    and after the end: every dt, the clock and the whole state."""
    kw = dict(gamma=1.4, limiter="VanLeer", riemann="HLLC", bc=bc, xmin=(0.2, 0, 0), xmax=(1.2, 1, 1))
    if geom == "Spherical":
        kw.update(gravity="Point_mass", central_mass=1e8)
    o = Oracle(1, [n], ng=ng, geom=geom, **kw)
    rho, rhou, E, fx = o.init_from_prim(*flow(o, n))
    d = Domain(1, [n], nghost=ng, geometry=geom, precision="fp64", **kw)
    d.set_state(rho, rhou, E)
    _, _, st, dts = o.run(rho, rhou, E, fx, cfl=0.3, max_iter=13, record_dts=True)
    assert st == 0
    d.run(cfl=0.3, nsteps=4)
    d.run(cfl=0.3, nsteps=9)
    assert np.array_equal(d.dt_log()[:13], dts)
    for a, ref in zip(d.get_state(), (rho, rhou, E)):
        assert np.array_equal(a, ref)
    t0 = float(np.sum(dts))
    d.set_state(rho, rhou, E)
    t, it, st, _ = o.run(rho, rhou, E, fx, cfl=0.3, t_end=0.1 * t0, max_iter=50, time_frequency=0.04 * t0)
    assert st == 0
    r = d.run(cfl=0.3, t_end=0.1 * t0, max_iter=50, time_frequency=0.04 * t0)
    assert (r.t, r.iter, r.finished) == (t, it, 1)
    for a, ref in zip(d.get_state(), (rho, rhou, E)):
        assert np.array_equal(a, ref)
