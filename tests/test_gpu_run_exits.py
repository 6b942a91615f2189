"""How a run of the FP64 step kernels ends, against the oracle: a state that
turns invalid after several steps, a time step that is not positive, an end
inside a launch of many steps, more steps than one launch of the 1-D cluster
holds, given time steps; on each route (1-D cluster, 2-D and 3-D marches,
tiles).  Also the cluster in the fast FP64 forms at the edges of its runs."""
import numpy as np
import pytest

from cases import rel_l1
from heraclespp_b200 import Domain, setups
from oracle import Oracle
from test_gpu_march64 import PHYS

pytestmark = pytest.mark.gpu
INVALID, NEGATIVE_DT = 4, 5
GRIDS = [[1000], [513], [330, 256], [100, 60], [60, 40, 60], [20, 18, 12]]


def streams(o, seed=3):
    rng = np.random.default_rng(seed)
    rho, u, P = setups.Grid.from_domain(o).alloc()
    rho[...] = 1 + 0.3 * rng.uniform(-1, 1, rho.shape)
    P[...] = 0.05 * (1 + 0.3 * rng.uniform(-1, 1, rho.shape))
    for d in range(o.ndim):
        u[d] = 0.6 * rng.uniform(-1, 1, rho.shape)
    return rho, u, P


def pair(nx, lim="VanLeer", rs="HLLC", precision="fp64", **kw):
    nd = len(nx)
    kw = dict(gamma=1.4, limiter=lim, riemann=rs, bc=["Periodic"] * (2 * nd)) | kw
    geom = kw.pop("geom", "Cartesian")
    o = Oracle(nd, nx, geom=geom, **kw)
    rho, rhou, E, fx = o.init_from_prim(*streams(o))
    d = Domain(nd, nx, geometry=geom, precision=precision, **kw)
    d.set_state(rho, rhou, E)
    u, P = o.conv_cons_to_prim(2, rho, rhou, E)
    return o, d, (rho, rhou, E, fx), 0.4 * o.time_step(2, rho, u, P)


def same_state(d, q):
    for a, ref in zip(d.get_state(), q[:3]):
        assert np.array_equal(a, ref, equal_nan=True)


@pytest.mark.parametrize("rs,lim", [("HLLC", "VanLeer"), ("HLL", "Minmod")])
@pytest.mark.parametrize("nx", GRIDS)
def test_state_turns_invalid(nx, rs, lim):
    """Time steps that grow by a fifth each: after 11 to 17 of them an internal
    energy is negative.  The run ends there, whatever was asked for."""
    o, d, q, dt0 = pair(nx, lim, rs)
    dts = dt0 * 1.2 ** np.arange(60)
    t, it, st, log = o.run(*q, max_iter=60, dts=dts, record_dts=True)
    assert st == 1 and 5 < it < 30
    rho, rhou, E = q[:3]
    with np.errstate(all="ignore"):
        evol = E - np.sum(rhou * rhou, axis=0) / rho / 2
    inner = np.zeros(E.shape, bool)
    inner[tuple(slice(2, -2) if n > 1 else slice(None) for n in E.shape)] = True
    first = int(np.flatnonzero((inner & ~(evol >= 0)).ravel())[0])
    r = d.run(nsteps=60, dts=dts, check_status=False)
    assert (r.status, r.iter, r.t, r.bad_cell) == (INVALID, it, t, first)
    assert np.array_equal(d.dt_log()[:it], log)
    same_state(d, q)


@pytest.mark.parametrize("nx", GRIDS)
def test_time_step_not_positive(nx):
    """An output time that has passed already asks for a negative step."""
    o, d, q, _ = pair(nx)
    t, it, st, log = o.run(*q, cfl=0.3, max_iter=4, record_dts=True)
    assert st == 0
    d.run(cfl=0.3, nsteps=4)
    assert o.run(*q, cfl=0.3, t_ini=t, max_iter=9, time_frequency=1.0, time_first_output=0.5 * t)[1:3] == (0, 2)
    r = d.run(cfl=0.3, nsteps=5, time_frequency=1.0, time_first_output=0.5 * t, check_status=False)
    assert (r.status, r.iter, r.t) == (NEGATIVE_DT, 4, t)
    assert np.array_equal(d.dt_log()[:4], log)
    same_state(d, q)


@pytest.mark.parametrize("nx", GRIDS)
def test_end_inside_a_launch(nx):
    """t_end is reached long before the number of steps asked for; a further run
    starts the loop again, whose first step has no time left."""
    o, d, q, dt0 = pair(nx)
    t, it, st, log = o.run(*q, cfl=0.3, t_end=5 * dt0, max_iter=50, record_dts=True)
    assert st == 0 and 3 < it < 40
    r = d.run(cfl=0.3, t_end=5 * dt0, nsteps=50)
    assert (r.status, r.iter, r.t, r.finished) == (0, it, t, 1)
    assert np.array_equal(d.dt_log()[:it], log)
    same_state(d, q)
    assert o.run(*q, cfl=0.3, t_ini=t, t_end=5 * dt0, max_iter=3)[:3] == (t, 1, 0)
    r = d.run(cfl=0.3, t_end=5 * dt0, nsteps=3)
    assert (r.status, r.iter, r.t) == (0, it + 1, t)
    same_state(d, q)


def test_more_steps_than_one_launch():
    o, d, q, _ = pair([48])
    t, it, st, log = o.run(*q, cfl=0.4, max_iter=5000, record_dts=True)
    assert (it, st) == (5000, 0)
    r = d.run(cfl=0.4, nsteps=5000)
    assert (r.status, r.iter, r.t) == (0, 5000, t)
    assert np.array_equal(d.dt_log()[:5000], log)
    same_state(d, q)


@pytest.mark.parametrize("geom,bc", [("Cartesian", ["Reflexive", "NullGradient"]), ("Spherical", ["Reflexive", "NullGradient"])])
@pytest.mark.parametrize("lim,rs", PHYS)
@pytest.mark.parametrize("n", [31, 33, 512, 513, 8192])
def test_fast_forms_in_the_cluster(n, lim, rs, geom, bc):
    o, d, q, dt0 = pair([n], lim, rs, "fp64_fast", geom=geom, bc=bc, xmin=(0.2, 0, 0), xmax=(1.2, 1, 1))
    dts = np.full(8, 0.5 * dt0)
    assert o.run(*q, max_iter=8, dts=dts)[1:3] == (8, 0)
    d.run(nsteps=8, dts=dts)
    for a, ref in zip(d.get_state(), q[:3]):
        assert rel_l1(a, ref) < 1e-12  # the bound of the fast FP64 tests
