"""The branch-free FP64 quotients and roots (csrc/quot64.cuh) against the
CPU's IEEE operators, bit for bit, through the stage entry points built on
them: states that cover every exponent, zeros, subnormals and the
significands the reciprocal iteration rounds wrongly, so that both the
straight-line path and the plain operators behind it are compared."""
import numpy as np
import pytest

from heraclespp_b200 import Domain
from oracle import Oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_conversions_over_all_exponents():
    """cons -> prim of states whose density, momenta and energy span the whole
    FP64 range: equal to the CPU's operators wherever the CPU's result is a
    number, and not a number where it is not."""
    nx = [96, 64]
    kw = dict(gamma=1.4, limiter="VanLeer", riemann="HLLC", bc=["Periodic"] * 4)
    o = Oracle(2, nx, **kw)
    rng = np.random.default_rng(3)
    shape = o.zeros().shape

    def wide(lo, hi):
        return np.ldexp(rng.uniform(1, 2, shape), rng.integers(lo, hi, shape))

    rho = wide(-1070, 1020)
    m = np.stack([wide(-1074, 500) * rng.choice([-1.0, 0.0, 1.0], shape) for _ in range(2)])
    E = wide(-1070, 1000)
    k = rng.random(shape)
    rho[k < 0.5] = rng.uniform(0.1, 10, np.count_nonzero(k < 0.5))
    E[k < 0.4] = rng.uniform(1, 10, np.count_nonzero(k < 0.4))
    ones = (k > 0.2) & (k < 0.3)  # significands of all ones
    rho[ones] = np.nextafter(np.ldexp(1.0, rng.integers(-3, 4, np.count_nonzero(ones))), 0.0)
    m[:, ones] = np.ldexp(1.0, rng.integers(-3, 4, (2, np.count_nonzero(ones))))
    u, P = o.conv_cons_to_prim(2, rho, m, E)
    d = Domain(2, nx, **kw)
    t = [torch.tensor(a, device="cuda") for a in (rho, m, E)]
    t += [torch.zeros_like(t[1]), torch.zeros_like(t[0])]
    d.conv_cons_to_prim(2, *t)
    torch.cuda.synchronize()
    for got, ref in ((t[3].cpu().numpy(), u), (t[4].cpu().numpy(), P)):
        assert np.array_equal(got, ref, equal_nan=True)
