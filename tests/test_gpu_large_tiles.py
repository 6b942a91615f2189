"""The FP64 2-D tile kernels on grids of more tiles than one wave holds, which
the smaller parity cases do not reach, against the oracle."""
import numpy as np
import pytest

from cases import oracle_kwargs, rel_l1
from heraclespp_b200 import Domain, setups
from oracle import Oracle

pytestmark = pytest.mark.gpu

WEDGE = dict(geometry="Spherical", xmin=(0.4, 0.6, 0.0), xmax=(1.4, 2.2, 1.0))
BC = ["Reflexive", "NullGradient", "Reflexive", "Periodic"]
RAD = dict(gamma=5.0 / 3.0, mmw=0.6, eos="RadGas")


def noise(o, seed, p0, v0):
    rng = np.random.default_rng(seed)
    rho, u, P = setups.Grid.from_domain(o).alloc()
    rho[...] = 1 + 0.3 * rng.uniform(-1, 1, rho.shape)
    P[...] = p0 * (1 + 0.3 * rng.uniform(-1, 1, rho.shape))
    u[...] = v0 * rng.uniform(-1, 1, u.shape)
    corner = np.s_[..., : rho.shape[-2] // 3, : rho.shape[-1] // 3]
    rho[corner], P[corner], u[corner] = 1.0, p0, 0.0
    fx = rng.uniform(0, 1, (o.nfx,) + rho.shape) if o.nfx else None
    return rho, u, P, fx


def run_both(nx, kw, nfx=0, steps=4, p0=1.0, v0=0.5, pressure_fix=False, precision="fp64", dts=None):
    ok = oracle_kwargs(kw)
    o = Oracle(2, nx, nfx=nfx, **ok)
    rho0, u0, P0, fx = noise(o, 11, p0, v0)
    rho, rhou, E, _ = o.init_from_prim(rho0, u0, P0)
    o.boundaries(rho, rhou, E, fx)
    d = Domain(2, nx, nfx=nfx, precision=precision, pressure_fix=pressure_fix, eps_pf=0.5, **kw)
    d.set_state(rho, rhou, E, fx=fx)
    _, it, st, dts = o.run(rho, rhou, E, fx, cfl=0.3, max_iter=steps, record_dts=True, pressure_fix=pressure_fix, eps_pf=0.5)
    assert (it, st) == (steps, 0)
    if precision == "fp64":
        d.run(cfl=0.3, nsteps=steps)
    else:
        d.run(nsteps=steps, dts=dts)
    got_fx = np.zeros_like(fx) if nfx else None
    got = d.get_state(fx=got_fx)
    pairs = list(zip(got, (rho, rhou, E))) + ([(got_fx, fx)] if nfx else [])
    return d.dt_log()[:steps], dts, pairs


@pytest.mark.parametrize("lim,rs", [("Minmod", "HLLC"), ("VanLeer", "HLL")])
@pytest.mark.parametrize("nx,nfx", [([300, 280], 0), ([161, 190], 0), ([300, 280], 1)])
def test_radgas(nx, nfx, lim, rs):
    """1e-12: CUDA's pow and the host's may round differently."""
    kw = dict(limiter=lim, riemann=rs, bc=BC, **RAD)
    log, dts, pairs = run_both(nx, kw, nfx, p0=1e13, v0=1e6)
    assert np.allclose(log, dts, rtol=1e-12, atol=0)
    for a, ref in pairs:
        assert rel_l1(a, ref) < 1e-12


# name: (grid arguments, nfx, pressure fix); 250 x 200 is 208 tiles of 16 x 16 and
# 300 x 280 is 342: one partial and more than one wave at two CTAs per SM
PERFECT = {
    "cartesian": (dict(g=(0.03, -0.05, 0.0)), 0, False),
    "spherical": (WEDGE, 0, False),
    "point mass": (dict(gravity="Point_mass", central_mass=1e8, **WEDGE), 0, False),
    "two scalars": (dict(), 2, False),
    "spherical scalar": (WEDGE, 1, False),
    "pressure fix": (dict(), 0, True),
}


@pytest.mark.parametrize("precision", ["fp64", "fp64_fast"])
@pytest.mark.parametrize("lim,rs", [("VanLeer", "HLLC"), ("Minmod", "HLL"), ("VanAlbada", "Low Mach")])
@pytest.mark.parametrize("name", PERFECT)
@pytest.mark.parametrize("nx", [[250, 200], [300, 280]])
def test_perfect_gas(nx, name, lim, rs, precision):
    extra, nfx, fix = PERFECT[name]
    kw = dict(gamma=1.4, limiter=lim, riemann=rs, bc=BC, **extra)
    log, dts, pairs = run_both(nx, kw, nfx, pressure_fix=fix, precision=precision)
    assert precision == "fp64_fast" or np.array_equal(log, dts)
    for a, ref in pairs:
        if precision == "fp64":
            assert np.array_equal(a, ref)
        else:
            assert rel_l1(a, ref) < 1e-12  # the bound of the fast FP64 tests


def stretched(nx, hi, ng=2):
    """Widths that vary smoothly by a factor of two; the ghost widths repeat the
    interior's."""
    nodes = []
    for n, h in zip(nx, hi):
        s = (np.arange(n + 2 * ng + 1) - ng) / n
        nodes.append(h * (s + 0.35 * np.sin(2 * np.pi * s) / (2 * np.pi)))
    return nodes + [np.array([0.0, 1.0])] * (3 - len(nx))


@pytest.mark.parametrize("precision", ["fp64", "fp64_fast"])
@pytest.mark.parametrize("lim,rs", [("VanLeer", "HLLC"), ("Minmod", "HLL"), ("VanAlbada", "Low Mach"), ("Constant", "HLLC")])
@pytest.mark.parametrize("nx", [[300, 280], [253, 310], [3, 4800]])
def test_march_on_user_defined_nodes(nx, lim, rs, precision):
    """The march divides by each column's and row's own widths."""
    kw = dict(gamma=1.4, limiter=lim, riemann=rs, bc=["NullGradient", "Reflexive", "Periodic", "Periodic"],
              nodes=stretched(nx, (1.0, 0.7)), xmax=(1.0, 0.7, 1.0), g=(0.03, -0.05, 0.0))
    log, dts, pairs = run_both(nx, kw, precision=precision)
    assert precision == "fp64_fast" or np.array_equal(log, dts)
    for a, ref in pairs:
        if precision == "fp64":
            assert np.array_equal(a, ref)
        else:
            assert rel_l1(a, ref) < 1e-12
