"""Every stage entry point of the FP64 path on operands out of the ordinary, bit
for bit against the oracle's plain operators: velocities over all exponents down
to subnormals and zeros, densities and pressures around the bounds of the shared
reciprocals (csrc/quot64.cuh: 2^-300 and 2^200) and far outside, significands of
all ones, and the denominators next to a power of two whose quotients lie next
to a midpoint.  This covers both the straight-line groups and what stands behind
them in the limiters, the face conversion, the Riemann solvers, the sound speed
and the time step."""
import numpy as np
import pytest

from cases import oracle_kwargs
from heraclespp_b200 import Domain, setups
from oracle import Oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SPH = dict(geometry="Spherical", xmin=(0.3, 0.6, 0.1), xmax=(1.0, 2.5, 1.5))
SHAPES = [([97], {}), ([40, 24], {}), ([18, 14, 10], {}), ([61], SPH), ([22, 18], SPH), ([12, 10, 8], SPH)]
KINDS = ["tiny", "subnormal", "low bound", "high bound", "scaled up", "scaled down", "ones"]
PHYS = [("VanLeer", "HLLC"), ("Minmod", "HLL"), ("VanAlbada", "HLLC"), ("Constant", "HLL"), ("Minmod", "Low Mach")]


def state(o, kind):
    rng = np.random.default_rng(len(kind) + 10 * o.ndim)
    rho, u, P = setups.Grid.from_domain(o).alloc()
    shape = rho.shape

    def sized(lo, hi, like):
        return np.ldexp(rng.uniform(1, 2, like.shape), rng.integers(lo, hi, like.shape)) * rng.choice([-1.0, 0.0, 1.0], like.shape)

    rho[...] = 1 + 0.3 * rng.uniform(-1, 1, shape)
    P[...] = 1 + 0.3 * rng.uniform(-1, 1, shape)
    u[...] = 0.5 * rng.uniform(-1, 1, u.shape)
    if kind == "tiny":
        u[...] = sized(-1022, 0, u)
    elif kind == "subnormal":
        u[...] = sized(-1074, -1015, u)
    elif kind.endswith("bound"):  # velocities around the numerators' bound, 2^-800 over the density, too
        f = np.ldexp(1.0, rng.integers(-304, -296, shape) if kind == "low bound" else rng.integers(196, 203, shape))
        rho *= f
        P *= f
        u[...] = np.where(rng.random(u.shape) < 0.5, sized(-505, -490, u) if kind == "low bound" else sized(-1005, -995, u), u)
    elif kind.startswith("scaled"):
        f = 2.0 ** (400 if kind == "scaled up" else -400)
        rho *= f
        P *= f
    else:
        rho[...] = np.where(rng.random(shape) < 0.5, np.nextafter(1.0, 0.0), 1.0)
        P[...] = np.where(rng.random(shape) < 0.5, np.nextafter(2.0, 0.0), 2.0)
        u[...] = np.where(rng.random(u.shape) < 0.5, 0.0, u)
    return rho, u, P


def dev(a):
    return torch.tensor(np.ascontiguousarray(a), device="cuda")


def host(t):
    torch.cuda.synchronize()
    return t.cpu().numpy()


def same(got, ref, what):
    got, ref = host(got).reshape(-1), np.asarray(ref).reshape(-1)
    wrong = ~((got == ref) | (np.isnan(got) & np.isnan(ref)))
    assert not wrong.any(), (what, np.count_nonzero(wrong), got[wrong][:3], ref[wrong][:3])


@pytest.mark.parametrize("lim,rs", PHYS)
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("nx,extra", SHAPES)
def test_stages(nx, extra, kind, lim, rs):
    nd = len(nx)
    kw = dict(gamma=1.4, limiter=lim, riemann=rs, bc=["Periodic"] * (2 * nd), **extra)
    o = Oracle(nd, nx, nfx=1, **oracle_kwargs(kw))
    d = Domain(nd, nx, nfx=1, **kw)
    rho, u, P = state(o, kind)
    fx = np.random.default_rng(1).uniform(0, 1, (1,) + rho.shape)
    with np.errstate(all="ignore"):
        rhou, E = o.conv_prim_to_cons(2, rho, u, P)
        u2, P2 = o.conv_cons_to_prim(2, rho, rhou, E)
        step = o.time_step(2, rho, u, P)
        dt = 0.3 * step
        rec = o.hydro_reconstruction(1, dt / 2, rho, u, P, fx)
        new = o.godunov(0, dt, rho, rhou, E, *rec[:3], fx, rec[3])
        evol = o.min_internal_energy(rho, rhou, E)
    t = [dev(a) for a in (rho, u, P, rhou, E, fx)]
    z = [torch.zeros_like(a) for a in t]
    d.conv_prim_to_cons(2, t[0], t[1], t[2], z[3], z[4])
    same(z[3], rhou, "rhou")
    same(z[4], E, "E")
    d.conv_cons_to_prim(2, t[0], t[3], t[4], z[1], z[2])
    same(z[1], u2, "u")
    same(z[2], P2, "P")
    same(torch.tensor([d.time_step(2, *t[:3]), d.minimum_internal_energy(t[0], *t[3:5])], dtype=torch.float64),
         [step, evol], "time step, internal energy")
    # face values of every variable, and the same from the whole reconstruction
    faces = {}
    for name, a in [("rho", rho), ("P", P), ("fx", fx[0])] + [(f"u{k}", u[k]) for k in range(nd)]:
        out = torch.zeros((nd, 2) + rho.shape, dtype=torch.float64, device="cuda")
        d.face_reconstruction(1, dev(a), out)
        faces[name] = o.face_reconstruction(1, np.ascontiguousarray(a))
        same(out, faces[name], "faces of " + name)
    g = [torch.zeros(a.shape, dtype=torch.float64, device="cuda") for a in rec]
    u_rec = torch.zeros((nd, nd, 2) + rho.shape, dtype=torch.float64, device="cuda")
    P_rec = torch.zeros((nd, 2) + rho.shape, dtype=torch.float64, device="cuda")
    d.hydro_reconstruction(1, dt / 2, t[0], t[1], t[2], t[5], *g, u_rec, P_rec)
    for a, ref, what in zip(g, rec, ("rho_rec", "rhou_rec", "E_rec", "fx_rec")):
        same(a, ref, what)
    same(P_rec, faces["P"], "P_rec")
    same(u_rec, np.stack([faces[f"u{k}"] for k in range(nd)]), "u_rec")
    got = [torch.zeros(a.shape, dtype=torch.float64, device="cuda") for a in new]
    d.godunov_scheme(0, dt, t[0], t[3], t[4], t[5], *[dev(a) for a in rec], *got)
    for a, ref, what in zip(got, new, ("rho", "rhou", "E", "fx")):
        same(a, ref, "new " + what)


def hard_pairs():
    """Denominators (2^53 - k) 2^-52, k odd to 2^14, with the numerators whose
    quotients lie 2^-54 / b above and below a midpoint M 2^-54 of two doubles:
    A 2^54 = B M +- 1."""
    num, den = [], []
    for k in range(1, 1 << 14, 2):
        B = (1 << 53) - k
        inv = pow(B, -1, 1 << 54)
        for M, s in (((1 << 54) - inv, 1), (inv, -1)):
            if M >= 1 << 53:
                A, rest = divmod(B * M + s, 1 << 54)
                assert rest == 0
                num.append(A)
                den.append(B)
    return np.ldexp(np.array(num, dtype=np.float64), -52), np.ldexp(np.array(den, dtype=np.float64), -52)


@pytest.mark.parametrize("shift", [-40, -1, 0, 7, 60])
def test_quotients_next_to_a_midpoint(shift):
    m, rho = hard_pairs()
    assert len(m) > 8000
    rho = np.ldexp(rho, shift)
    nx = [128, 128]
    o = Oracle(2, nx, gamma=1.4)
    shape = o.zeros().shape
    R = np.ones(shape)
    M = np.zeros((2,) + shape)
    R.reshape(-1)[: len(rho)] = rho
    M[0].reshape(-1)[: len(m)] = m
    M[1].reshape(-1)[: len(m)] = -np.ldexp(m, 3)
    E = np.full(shape, 1e4) * np.maximum(R, 1 / R)
    u, P = o.conv_cons_to_prim(2, R, M, E)
    assert np.array_equal(u[0], M[0] / R)
    t = [dev(a) for a in (R, M, E)]
    out = [torch.zeros_like(t[1]), torch.zeros_like(t[0])]
    Domain(2, nx, gamma=1.4).conv_cons_to_prim(2, *t, *out)
    same(out[0], u, "u")
    same(out[1], P, "P")
