"""FP64 steps of gas at rest: a front runs into it, and ahead of the front the
velocities fall by orders of magnitude per cell through the smallest numbers to
exact zeros, densities lie one unit in the last place below 1, and the rest is
uniform.  Every such value must come out as the oracle's, bit for bit, on each
route (1-D cluster, 2-D and 3-D marches, tiles), and must not slow a step down."""
import numpy as np
import pytest

from heraclespp_b200 import Domain, setups
from oracle import Oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

GRIDS = [([700], 150), ([112, 96], 60), ([330, 256], 40), ([66, 31, 24], 16), ([20, 18, 12], 16)]
PHYS = [("VanLeer", "HLLC"), ("Minmod", "HLL"), ("VanAlbada", "HLLC"), ("Minmod", "Low Mach")]


def blast(o, rho0=1.0):
    rho, u, P = setups.Grid.from_domain(o).alloc()
    rho[...], P[...] = rho0, 1.0
    n = rho.shape
    P[tuple(slice(m // 2 - 3, m // 2 + 2) if m > 8 else slice(None) for m in n)] = 20.0
    return rho, u, P


def compare(o, nd, nx, prim, steps, ng=2, **kw):
    rho, rhou, E, fx = o.init_from_prim(*prim)
    start = (rho.copy(), rhou.copy(), E.copy())
    _, it, st, dts = o.run(rho, rhou, E, fx, cfl=0.4, max_iter=steps, record_dts=True)
    d = Domain(nd, nx, nghost=ng, precision="fp64", **kw)
    d.set_state(*start)
    r = d.run(cfl=0.4, nsteps=steps, check_status=False)
    # some slopes of subnormal numbers are not numbers (infinity over infinity):
    # the run stops there, as the oracle's does
    assert (r.iter, r.status) == (it, 4 if st == 1 else 0)
    assert np.array_equal(d.dt_log()[:it], dts)
    for a, ref in zip(d.get_state(), (rho, rhou, E)):
        assert np.array_equal(a, ref, equal_nan=True)
    return rhou


@pytest.mark.parametrize("lim,rs", PHYS)
@pytest.mark.parametrize("nx,steps", GRIDS)
def test_front_into_still_gas(nx, steps, lim, rs):
    nd = len(nx)
    kw = dict(gamma=1.4, limiter=lim, riemann=rs, bc=["NullGradient"] * (2 * nd))
    o = Oracle(nd, nx, **kw)
    m = np.abs(compare(o, nd, nx, blast(o), steps, **kw))
    assert np.any(m == 0)
    assert nd == 1 or np.any((m > 0) & (m < 1e-30))  # in 1-D two cells in one of the steps


@pytest.mark.parametrize("nx", [[700], [330, 256], [66, 31, 24], [100, 60]])
@pytest.mark.parametrize("what", ["u1e-120", "u1e-300", "u_subnormal", "2^400", "2^-400", "ulp"])
@pytest.mark.parametrize("lim,rs", PHYS[:3])
def test_values_of_every_size(nx, what, lim, rs):
    """Velocities of one tiny size in half of the domain; a flow whose density
    and pressure are scaled out of the shared reciprocals' range; densities a
    unit in the last place below 1."""
    nd = len(nx)
    kw = dict(gamma=1.4, limiter=lim, riemann=rs, bc=["Periodic"] * (2 * nd))
    o = Oracle(nd, nx, **kw)
    rng = np.random.default_rng(7)
    rho, u, P = setups.Grid.from_domain(o).alloc()
    rho[...] = 1 + 0.3 * rng.uniform(-1, 1, rho.shape)
    P[...] = 1 + 0.3 * rng.uniform(-1, 1, rho.shape)
    u[...] = 0.5 * rng.uniform(-1, 1, u.shape)
    half = np.s_[..., : rho.shape[-1] // 2]
    if what.startswith("u"):
        rho[half], P[half] = 1.0, 1.0
        if what == "ulp":
            rho[half] = np.where(rng.random(rho[half].shape) < 0.5, np.nextafter(1.0, 0.0), 1.0)
            u[half] = 0.0
        else:
            size = dict(zip(["u1e-120", "u1e-300", "u_subnormal"], [1e-120, 1e-300, 1e-310]))[what]
            u[half] *= size
    else:
        f = 2.0 ** int(what[2:])
        rho *= f
        P *= f
    compare(o, nd, nx, (rho, u, P), 4, **kw)


def us_per_step(d, prim, steps):
    s = torch.cuda.ExternalStream(d.stream_handle())
    best = np.inf
    for _ in range(5):
        d.set_state_from_prim(*prim)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(s)
        d.run(cfl=0.4, nsteps=steps)
        e1.record(s)
        e1.synchronize()
        best = min(best, e0.elapsed_time(e1) / steps * 1e3)
    return best


@pytest.mark.parametrize("prec", ["fp64", "fp64_fast"])
@pytest.mark.parametrize("lim,rs,limit", [("Minmod", "HLL", 1.25), ("VanLeer", "HLLC", 1.8)])
def test_still_gas_costs_no_more(prec, lim, rs, limit):
    """A blast in still gas against noise in every cell, same grid, by device
    time.  A zero difference or momentum needs no second look (limit: the
    spread of timings); the few rows that a front's decaying tail crosses are
    done again out of line, and a strip of rows waits for them."""
    nx = [512, 512]
    kw = dict(gamma=1.4, limiter=lim, riemann=rs, bc=["NullGradient"] * 4)
    d = Domain(2, nx, precision=prec, **kw)
    still = blast(d)
    rng = np.random.default_rng(3)
    noise = [base + 0.1 * rng.uniform(-1, 1, a.shape) for base, a in zip((1.0, 0.0, 1.0), still)]
    assert us_per_step(d, still, 60) < limit * us_per_step(d, noise, 60)
