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
