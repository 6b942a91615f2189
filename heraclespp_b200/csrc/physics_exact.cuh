// physics_exact.cuh -- per-cell physics with the reference's FP64 arithmetic.
//
// Each function keeps the association order of the reference expression it
// restates, and the translation units that include this header are built
// with --fmad=false, so the device results round exactly like the reference's
// FP64 CPU build: every quotient and square root is the rounded one, formed
// from shared reciprocals (quot64.cuh) or, out of their range, by IEEE
// division and square root.  State vectors are [rho, v_0..v_{ND-1}, E or P].
//
// Eos kind EOS_PERFECT_GAS_FAST selects the fast-FP64 forms instead (used by
// the fused kernels of the fast-FP64 precision, built with FMA contraction):
// the same mathematics with fewer divisions -- P = (gamma-1) e and
// e = P/(gamma-1) (the temperature factors of perfect_gas.hpp:46-83 cancel),
// one reciprocal of rho per state, limiters on raw differences
// (slope_limiters.hpp:38-85: van Leer 2RL/(R+L), minmod the smaller of R and
// L, van Albada RL(R+L)/(R^2+L^2)) and one reciprocal of S - u* in HLLC.
// Results differ from the reference by rounding only (~1e-16 per operation).
#pragma once

#include "hcl_device.cuh"
#include "quot64.cuh"

namespace hcl::exact {

struct Eos {
    double gamma, gamma_m1, mmw;
    int kind; // EOS_PERFECT_GAS, EOS_RAD_GAS or EOS_PERFECT_GAS_FAST
    // the perfect gas's constant denominators (perfect_gas.hpp:46-83): mu m_p
    // and mu m_p (gamma - 1); consts_ok: both usable as such, and the internal
    // energy not far below the pressure
    q64::Den mk, ev;
    bool consts_ok;
};

__device__ __forceinline__ Eos make_eos(double gamma, double gamma_m1, double mmw, int kind)
{
    const double b = mmw * kMp;
    const double c = mmw * kMp * gamma_m1;
    return Eos{gamma, gamma_m1, mmw, kind, q64::Den{b, 1.0 / b}, q64::Den{c, 1.0 / c},
               q64::den_ok(b) && q64::den_ok(c) && gamma_m1 <= 1024.0};
}

__device__ __forceinline__ Eos eos_of(const GridDev& g)
{
    return make_eos(g.gamma, g.gamma_m1, g.mmw, g.eos);
}

// thermodynamics/rad_gas.hpp:47-146: gas plus radiation.  The temperature
// comes from a Newton iteration (at most 100 steps, stop at |dT| <= 1e-6)
// started at the larger of the gas-only and radiation-only temperatures.
namespace rad {
__device__ __forceinline__ double evol_from_temp(const Eos& e, double rho, double T)
{
    const double T4 = T * T * T * T;
    return (rho * kKb * T / (e.mmw * kMp * e.gamma_m1)) + (kAr * T4);
}
__device__ __forceinline__ double pres_from_temp(const Eos& e, double rho, double T)
{
    const double T4 = T * T * T * T;
    return (rho * kKb * T / (e.mmw * kMp)) + (kAr * T4 / 3);
}
static __device__ __noinline__ double temp_from_pres(const Eos& e, double rho, double P)
{
    const double C1 = rho * kKb / (e.mmw * kMp);
    const double Tg = P / C1;
    const double Tr = pow(3 * P / kAr, 1. / 4);
    double T = Tr > Tg ? Tr : Tg;
    for (int i = 0; i < 100; ++i) {
        const double T3 = T * T * T;
        const double f = (kAr * T3 * T / 3) + (C1 * T) - P;
        const double df = (4 * kAr * T3 / 3) + C1;
        const double delta_T = -f / df;
        T += delta_T;
        if (fabs(delta_T) <= 1E-6) {
            break;
        }
    }
    return T;
}
static __device__ __noinline__ double temp_from_evol(const Eos& e, double rho, double evol)
{
    const double C1 = rho * kKb / (e.mmw * kMp * e.gamma_m1);
    const double Tg = evol / C1;
    const double Tr = pow(evol / kAr, 1. / 4);
    double T = Tr > Tg ? Tr : Tg;
    for (int i = 0; i < 100; ++i) {
        const double T3 = T * T * T;
        const double f = (kAr * T3 * T) + (C1 * T) - evol;
        const double df = (4 * kAr * T3) + C1;
        const double delta_T = -f / df;
        T += delta_T;
        if (fabs(delta_T) <= 1E-6 || isnan(delta_T)) {
            break;
        }
    }
    return T;
}
static __device__ __noinline__ double sound(const Eos& e, double rho, double P)
{
    const double T = temp_from_pres(e, rho, P);
    const double Pg = rho * kKb * T / (e.mmw * kMp);
    const double T4 = T * T * T * T;
    const double Pr = kAr * T4 / 3;
    const double alpha = Pr / Pg;
    const double num = (e.gamma / (e.gamma - 1)) + (20 * alpha) + (16 * alpha * alpha);
    const double den = (1. / (e.gamma - 1)) + (12 * alpha);
    const double gamma_eff = num / den;
    return sqrt(gamma_eff * Pg / rho);
}
} // namespace rad

// thermodynamics/perfect_gas.hpp:46-83: P <-> e through the temperature.
__device__ __forceinline__ double temp_from_pres(const Eos& e, double rho, double P)
{
    return P * e.mmw * kMp / (rho * kKb);
}
__device__ __forceinline__ double evol_from_temp(const Eos& e, double rho, double T)
{
    return rho * kKb * T / (e.mmw * kMp * e.gamma_m1);
}
__device__ __forceinline__ double pres_from_temp(const Eos& e, double rho, double T)
{
    return rho * kKb * T / (e.mmw * kMp);
}
__device__ __forceinline__ double temp_from_evol(const Eos& e, double rho, double evol)
{
    return evol * e.mmw * kMp * e.gamma_m1 / (rho * kKb);
}
// compute_temp_from_pres of the configured EOS (perfect_gas.hpp:64-68,
// rad_gas.hpp:71-89)
__device__ __forceinline__ double temperature(const Eos& e, double rho, double P)
{
    if (e.kind == EOS_RAD_GAS) {
        return rad::temp_from_pres(e, rho, P);
    }
    return temp_from_pres(e, rho, P);
}
__device__ __forceinline__ double evol_from_pres(const Eos& e, double rho, double P)
{
    if (e.kind == EOS_PERFECT_GAS_FAST) {
        return P * (1.0 / e.gamma_m1);
    }
    if (e.kind == EOS_RAD_GAS) {
        return rad::evol_from_temp(e, rho, rad::temp_from_pres(e, rho, P)); // rad_gas.hpp:47-51
    }
    return evol_from_temp(e, rho, temp_from_pres(e, rho, P));
}
__device__ __forceinline__ double pres_from_evol(const Eos& e, double rho, double evol)
{
    if (e.kind == EOS_PERFECT_GAS_FAST) {
        return e.gamma_m1 * evol;
    }
    if (e.kind == EOS_RAD_GAS) {
        return rad::pres_from_temp(e, rho, rad::temp_from_evol(e, rho, evol)); // rad_gas.hpp:65-69
    }
    return pres_from_temp(e, rho, temp_from_evol(e, rho, evol));
}
__device__ __forceinline__ double plain_sound(const Eos& e, double rho, double P)
{
    if (e.kind == EOS_RAD_GAS) {
        return rad::sound(e, rho, P);
    }
    return sqrt(e.gamma * P / rho);
}

// The step's algebra with the plain operators: what every fast form below
// falls back to when an operand is near overflow or underflow, the RadGas
// path, and the low-Mach solver's own expressions.
namespace plain {
// hydro/euler_equations.hpp:41-59
template <int ND>
__device__ __forceinline__ double ek_cons(const double* c)
{
    double norm = 0;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        norm += c[1 + d] * c[1 + d];
    }
    return norm / c[0] / 2;
}
template <int ND>
__device__ __forceinline__ double ek_prim(const double* p)
{
    double norm = 0;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        norm += p[1 + d] * p[1 + d];
    }
    return p[0] * norm / 2;
}

// hydro/euler_equations.hpp:111-122
template <int ND>
__device__ __forceinline__ void to_prim(const Eos& e, const double* c, double* p)
{
    if (e.kind == EOS_PERFECT_GAS_FAST) {
        const double ir = 1.0 / c[0];
        double mu = 0;
        p[0] = c[0];
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            p[1 + d] = c[1 + d] * ir;
            mu += c[1 + d] * p[1 + d];
        }
        p[1 + ND] = e.gamma_m1 * (c[1 + ND] - 0.5 * mu);
        return;
    }
    const double evol = c[1 + ND] - ek_cons<ND>(c);
    p[0] = c[0];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        p[1 + d] = c[1 + d] / c[0];
    }
    p[1 + ND] = pres_from_evol(e, c[0], evol);
}

// hydro/euler_equations.hpp:124-134
template <int ND>
__device__ __forceinline__ void to_cons(const Eos& e, const double* p, double* c)
{
    c[0] = p[0];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        c[1 + d] = p[0] * p[1 + d];
    }
    c[1 + ND] = evol_from_pres(e, p[0], p[1 + ND]) + ek_prim<ND>(p);
}

// hydro/euler_equations.hpp:72-86
template <int ND>
__device__ __forceinline__ void flux_prim(const Eos& e, const double* p, int l, double* f)
{
    const double P = p[1 + ND];
    const double E = ek_prim<ND>(p) + evol_from_pres(e, p[0], P);
    f[0] = p[0] * p[1 + l];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        f[1 + d] = p[0] * p[1 + l] * p[1 + d];
    }
    f[1 + l] += P;
    f[1 + ND] = p[1 + l] * (E + P);
}

// hydro/slope_limiters.hpp:18-87 (division forms kept as written; the
// raw-difference forms for kind EOS_PERFECT_GAS_FAST)
__device__ __forceinline__ double slope(int lim, double diffR, double diffL, int kind = EOS_PERFECT_GAS)
{
    if (lim == LIM_CONSTANT) {
        return 0;
    }
    if (kind == EOS_PERFECT_GAS_FAST) {
        const double prod = diffR * diffL;
        if (!(prod > 0)) {
            return 0;
        }
        if (lim == LIM_VANLEER) {
            return 2 * prod / (diffR + diffL);
        }
        if (lim == LIM_MINMOD) {
            return fabs(diffR) < fabs(diffL) ? diffR : diffL;
        }
        return prod * (diffR + diffL) / (diffR * diffR + diffL * diffL);
    }
    if (diffL * diffR > 0) {
        const double ratio = diffR / diffL;
        if (lim == LIM_VANLEER) {
            return (1. / 2) * (diffR + diffL) * (4 * ratio) / ((ratio + 1) * (ratio + 1));
        }
        if (lim == LIM_MINMOD) {
            const double minmod = 2 * fmin(1., ratio) / (1 + ratio);
            return minmod * (diffL + diffR) / 2;
        }
        return (1. / 2) * (diffR + diffL) * (2 * ratio) / ((ratio * ratio) + 1);
    }
    return 0;
}

// hydro/riemann_solver.hpp:60-64, :136-140
__device__ __forceinline__ double flux_hll(double UL, double UR, double FL, double FR, double wsL, double wsR)
{
    return ((wsR * FL) - (wsL * FR) + (wsL * wsR * (UR - UL))) / (wsR - wsL);
}
__device__ __forceinline__ double flux_hllc(double F, double U, double Ustar, double ws)
{
    return F + (ws * (Ustar - U));
}

// hydro/riemann_solver.hpp:22-181.  cL/cR: conservative states; l: direction.
template <int ND>
__device__ __forceinline__ void riemann(const Eos& e, int solver, const double* cL, const double* cR, int l, double* f)
{
    double pL[ND + 2], pR[ND + 2];
    plain::to_prim<ND>(e, cL, pL);
    plain::to_prim<ND>(e, cR, pR);
    const double PL = pL[1 + ND];
    const double PR = pR[1 + ND];
    const double aL = plain_sound(e, pL[0], PL);
    const double aR = plain_sound(e, pR[0], PR);
    const double uL = pL[1 + l];
    const double uR = pR[1 + l];
    if (solver == RS_SPLITTING) {
        // :146-180
        const double a = 1.1 * fmax(pL[0] * aL, pR[0] * aR);
        const double ustar = ((uL + uR) / 2) - (1 / (2 * a) * (PR - PL));
        const double Ma = fabs(ustar) / fmin(aL, aR);
        const double theta = fmin(1., Ma);
        const double Pstar = ((PL + PR) / 2) - ((theta * a) / 2 * (uR - uL));
        const double* cs = (ustar > 0) ? cL : cR;
        f[0] = ustar * cs[0];
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            f[1 + d] = ustar * cs[1 + d];
        }
        f[1 + l] += Pstar;
        f[1 + ND] = (ustar * cs[1 + ND]) + (Pstar * ustar);
        return;
    }
    const double wsL = fmin(uL - aL, uR - aR);
    const double wsR = fmax(uL + aL, uR + aR);
    double fL[ND + 2], fR[ND + 2];
    plain::flux_prim<ND>(e, pL, l, fL);
    plain::flux_prim<ND>(e, pR, l, fR);
    if (solver == RS_HLL) {
        // :31-58
        const double neg_wsL = fmin(wsL, 0.);
        const double pos_wsR = fmax(wsR, 0.);
#pragma unroll
        for (int v = 0; v < ND + 2; ++v) {
            f[v] = flux_hll(cL[v], cR[v], fL[v], fR[v], neg_wsL, pos_wsR);
        }
        return;
    }
    // HLLC :70-134
    const double rcL = pL[0] * (wsL - uL);
    const double rcR = pR[0] * (wsR - uR);
    const double ustar = (PR - PL + (rcL * uL) - (rcR * uR)) / (rcL - rcR);
    const double pstar = 1. / 2 * (PL + PR + (rcL * (ustar - uL)) + (rcR * (ustar - uR)));
    const bool left = ustar > 0;
    const double S = left ? wsL : wsR;
    const double* cs = left ? cL : cR;
    const double* ps = left ? pL : pR;
    const double* fs = left ? fL : fR;
    const double un = ps[1 + l];
    if (wsL * wsR > 0) {
#pragma unroll
        for (int v = 0; v < ND + 2; ++v) {
            f[v] = fs[v];
        }
        return;
    }
    if (e.kind == EOS_PERFECT_GAS_FAST) {
        const double inv = 1.0 / (S - ustar);
        const double ratio = (S - un) * inv;
        const double rs = cs[0] * ratio;
        f[0] = flux_hllc(fs[0], cs[0], rs, S);
        const double rsu = rs * ustar;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            f[1 + d] = rsu * ps[1 + d];
        }
        f[1 + l] = rsu * ustar + pstar;
        const double Es = ratio * cs[1 + ND] + (ustar - un) * inv * (ustar * cs[0] * (S - un) + ps[1 + ND]);
        f[1 + ND] = flux_hllc(fs[1 + ND], cs[1 + ND], Es, S);
        return;
    }
    const double rho_star = cs[0] * (S - un) / (S - ustar);
    f[0] = flux_hllc(fs[0], cs[0], rho_star, S);
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        f[1 + d] = rho_star * ustar * ps[1 + d];
    }
    f[1 + l] = (rho_star * ustar * ustar) + pstar;
    const double E_star = ((S - un) / (S - ustar) * cs[1 + ND]) + ((ustar - un) / (S - ustar) * ((ustar * cs[0] * (S - un)) + ps[1 + ND]));
    f[1 + ND] = flux_hllc(fs[1 + ND], cs[1 + ND], E_star, S);
}
} // namespace plain

// hydro/euler_equations.hpp:41-59
using plain::ek_cons;

// ---- the same results with shared reciprocals (quot64.cuh) ------------------
// Each *_core evaluates a group of expressions straight through and gathers
// its operands in a range S: denominators, pressures, and numerators, which may
// be zero or smaller.  Where it holds every quotient and root is the rounded
// one.  Otherwise the group is done again out of line: with quo_tiny() for the
// numerators (TINY; the reference's arithmetic only) if those were the matter, else
// with plain operators.  Scalings by powers of two (the /2 of the kinetic
// energy, the 4/2 and 2/2 of the limiters) are folded, which is exact in that
// range.
template <int ND>
static __device__ __noinline__ void to_cons_flux_slow(Eos e, const double* p, int l, double* c, double* f)
{
    plain::to_cons<ND>(e, p, c);
    plain::flux_prim<ND>(e, p, l, f);
}
static __device__ __noinline__ double sound_slow(Eos e, double rho, double P)
{
    return plain_sound(e, rho, P);
}
// a numerator's quotient
template <bool TINY>
__device__ __forceinline__ double num_quo(double a, const q64::Den& d, q64::Range& S)
{
    if constexpr (TINY) {
        bool good = true;
        const double q = q64::quo_tiny(a, d, good);
        S.also(good);
        return q;
    } else {
        return q64::quo(a, d);
    }
}

// hydro/euler_equations.hpp:111-122.  r, k: the denominators rho and rho kb;
// evol: the internal energy.  S holds rho, P and the momenta.
template <int ND, bool TINY = false>
__device__ __forceinline__ void prim_core(const Eos& e, const double* c, double* p, q64::Den& r, q64::Den& k,
                                          double& evol, q64::Range& S)
{
    p[0] = c[0];
    if (e.kind == EOS_PERFECT_GAS_FAST) {
        r = q64::den(c[0]);
        double mu = 0;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            p[1 + d] = c[1 + d] * r.y;
            mu += c[1 + d] * p[1 + d];
        }
        evol = c[1 + ND] - 0.5 * mu;
        p[1 + ND] = e.gamma_m1 * evol;
        S.pos(c[0], p[1 + ND]);
        return;
    }
    r = q64::den(c[0]);
    double norm = 0;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        norm += c[1 + d] * c[1 + d];
        p[1 + d] = num_quo<TINY>(c[1 + d], r, S);
    }
    evol = __fma_rn(-0.5, q64::quo(norm, r), c[1 + ND]);
    const double kb = c[0] * kKb;
    k = q64::den_from(kb, r.y * (1 / kKb));
    p[1 + ND] = q64::quo(kb * q64::quo(evol * e.mmw * kMp * e.gamma_m1, k), e.mk);
    S.pos(c[0], p[1 + ND]);
    S.low(kb);
    S.num(c[1], c[ND >= 2 ? 2 : 1]);
    if constexpr (ND == 3) {
        S.num(c[3], c[3]);
    }
}
template <int ND, int KIND>
static __device__ __noinline__ void to_prim_slow(Eos e, const double* c, double* p)
{
    e.kind = KIND;
    if constexpr (KIND == EOS_PERFECT_GAS) {
        q64::Den r, k;
        double evol;
        q64::Range S(e.consts_ok);
        prim_core<ND, true>(e, c, p, r, k, evol, S);
        if (S.dens_ok()) {
            return;
        }
    }
    plain::to_prim<ND>(e, c, p);
}
template <int ND>
__device__ __forceinline__ void to_prim(const Eos& e, const double* c, double* p)
{
    if (e.kind == EOS_RAD_GAS) {
        plain::to_prim<ND>(e, c, p);
        return;
    }
    q64::Den r, k;
    double evol;
    q64::Range S(e.consts_ok);
    prim_core<ND>(e, c, p, r, k, evol, S);
    if (!S.ok()) {
        double ct[ND + 2], pt[ND + 2];
#pragma unroll
        for (int v = 0; v < ND + 2; ++v) {
            ct[v] = c[v];
        }
        if (e.kind == EOS_PERFECT_GAS_FAST) {
            to_prim_slow<ND, EOS_PERFECT_GAS_FAST>(e, ct, pt);
        } else {
            to_prim_slow<ND, EOS_PERFECT_GAS>(e, ct, pt);
        }
#pragma unroll
        for (int v = 0; v < ND + 2; ++v) {
            p[v] = pt[v];
        }
    }
}

// e(rho, P) of the perfect gas through the temperature; k: the denominator
// rho kb (perfect_gas.hpp:46-83).  In range where rho and P are.
__device__ __forceinline__ double evol_core(const Eos& e, double P, const q64::Den& k)
{
    return q64::quo(k.b * q64::quo(P * e.mmw * kMp, k), e.ev);
}

// hydro/euler_equations.hpp:124-134 and :72-86: the conservative state of a
// face and its flux along l, which share rho u_l and E
template <int ND>
__device__ __forceinline__ void cons_flux_core(const Eos& e, const double* p, int l, double* c, double* f, q64::Range& S)
{
    double evol;
    if (e.kind == EOS_PERFECT_GAS_FAST) {
        evol = p[1 + ND] * (1.0 / e.gamma_m1);
    } else {
        const double kb = p[0] * kKb;
        S.pos(p[0], p[1 + ND]);
        evol = evol_core(e, p[1 + ND], q64::den(kb));
    }
    double norm = 0;
    c[0] = p[0];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        c[1 + d] = p[0] * p[1 + d];
        norm += p[1 + d] * p[1 + d];
    }
    c[1 + ND] = __fma_rn(0.5, p[0] * norm, evol);
    f[0] = c[1 + l];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        f[1 + d] = c[1 + l] * p[1 + d];
    }
    f[1 + l] += p[1 + ND];
    f[1 + ND] = p[1 + l] * (c[1 + ND] + p[1 + ND]);
}

template <int ND>
__device__ __forceinline__ void to_cons_flux(const Eos& e, const double* p, int l, double* c, double* f)
{
    if (e.kind == EOS_RAD_GAS) {
        plain::to_cons<ND>(e, p, c);
        plain::flux_prim<ND>(e, p, l, f);
        return;
    }
    q64::Range S(e.consts_ok);
    cons_flux_core<ND>(e, p, l, c, f, S);
    if (!S.ok()) {
        double pt[ND + 2], ct[ND + 2], ft[ND + 2];
#pragma unroll
        for (int v = 0; v < ND + 2; ++v) {
            pt[v] = p[v];
        }
        to_cons_flux_slow<ND>(e, pt, l, ct, ft);
#pragma unroll
        for (int v = 0; v < ND + 2; ++v) {
            c[v] = ct[v];
            f[v] = ft[v];
        }
    }
}
template <int ND>
__device__ __forceinline__ void to_cons(const Eos& e, const double* p, double* c)
{
    double f[ND + 2];
    to_cons_flux<ND>(e, p, 0, c, f);
}
__device__ __forceinline__ double sound(const Eos& e, double rho, double P)
{
    if (e.kind == EOS_RAD_GAS) {
        return plain_sound(e, rho, P);
    }
    if (!(q64::den_ok(rho) && q64::within(P))) {
        return sound_slow(e, rho, P);
    }
    return q64::root(q64::quo(e.gamma * P, q64::den(rho)));
}

// What the health check and the CFL need of a new state: the internal energy
// (main.cpp:397-425), the primitives and the sound speed (time_step.hpp:55-77).
template <int ND, bool TINY = false>
__device__ __forceinline__ bool state_core(const Eos& e, const double* q, double& evol, double& snd, double* p)
{
    q64::Den r, k;
    q64::Range S(e.consts_ok);
    prim_core<ND, TINY>(e, q, p, r, k, evol, S);
    snd = q64::root(q64::quo(e.gamma * p[1 + ND], r));
    return TINY ? S.dens_ok() : S.ok();
}
template <int ND, int KIND>
static __device__ __noinline__ void state_prims_slow(Eos e, const double* q, double* out)
{
    e.kind = KIND;
    if constexpr (KIND == EOS_PERFECT_GAS) {
        if (state_core<ND, true>(e, q, out[0], out[1], out + 2)) {
            return;
        }
    }
    out[0] = q[1 + ND] - plain::ek_cons<ND>(q);
    plain::to_prim<ND>(e, q, out + 2);
    out[1] = plain_sound(e, out[2], out[3 + ND]);
}
template <int ND>
__device__ __forceinline__ void state_prims(const Eos& e, const double* q, double& evol, double& snd, double* p)
{
    if (e.kind == EOS_RAD_GAS || !state_core<ND>(e, q, evol, snd, p)) {
        double qt[ND + 2], ot[ND + 4];
#pragma unroll
        for (int v = 0; v < ND + 2; ++v) {
            qt[v] = q[v];
        }
        if (e.kind == EOS_PERFECT_GAS_FAST) {
            state_prims_slow<ND, EOS_PERFECT_GAS_FAST>(e, qt, ot);
        } else if (e.kind == EOS_RAD_GAS) {
            state_prims_slow<ND, EOS_RAD_GAS>(e, qt, ot);
        } else {
            state_prims_slow<ND, EOS_PERFECT_GAS>(e, qt, ot);
        }
        evol = ot[0];
        snd = ot[1];
#pragma unroll
        for (int v = 0; v < ND + 2; ++v) {
            p[v] = ot[2 + v];
        }
    }
}

// hydro/slope_limiters.hpp:18-87 on the two one-sided quotients: limited_core
// returns the slope, halved for van Leer (4 ratio / 2 folded), so that a face
// lies limited_core * limited_width from the centre.  FAST: the raw-difference
// forms.
template <int LIM>
__device__ __forceinline__ double limited_width(double dl)
{
    return LIM == LIM_VANLEER ? dl : dl / 2;
}
// S holds the quotients and the limiter's own denominator where their product
// is positive (or not a number): elsewhere the slope is zero whatever they are.
template <int LIM>
__device__ __forceinline__ double limited_den(double ratio)
{
    return LIM == LIM_VANLEER ? (ratio + 1) * (ratio + 1) : (LIM == LIM_MINMOD ? 1 + ratio : (ratio * ratio) + 1);
}
template <int LIM>
__device__ __forceinline__ double limited_core(double dR, double dL, q64::Range& S)
{
    const bool use = !(dL * dR <= 0);
    const double ratio = q64::quo(dR, q64::den(dL));
    const double b = limited_den<LIM>(ratio);
    const double num = LIM == LIM_MINMOD ? fmin(1., ratio) : (dR + dL) * ratio;
    double s = q64::quo(num, q64::den(b));
    if constexpr (LIM == LIM_MINMOD) {
        s = s * (dL + dR);
    }
    S.slope(use, dR, dL, b);
    S.low(dL);
    return use ? s : 0.0;
}
// The same for quotients down to 2^-1000 of one sign, tiny pairs scaled by a power
// of two (the slope scales with them); good turns false beyond that.
template <int LIM>
__device__ __forceinline__ double limited_tiny(double dR, double dL, bool& good)
{
    const double lo = fmin(fabs(dR), fabs(dL));
    const double hi = fmax(fabs(dR), fabs(dL));
    const bool use = !(dL * dR <= 0);
    const double up = lo < 0x1p-700 ? 0x1p400 : 1.0;
    const double down = lo < 0x1p-700 ? 0x1p-400 : 1.0;
    const double R = fabs(dR) * up, L = fabs(dL) * up;
    const double ratio = q64::quo(R, q64::den(L));
    const double b = limited_den<LIM>(ratio);
    const double num = LIM == LIM_MINMOD ? fmin(1., ratio) : (R + L) * ratio;
    double s = q64::quo(num, q64::den(b));
    if constexpr (LIM == LIM_MINMOD) {
        s = s * (L + R);
    }
    good = !use || (lo >= 0x1p-1000 && hi <= 0x1p200 && ratio >= 0x1p-1000 && ratio <= 0x1p400);
    return use ? copysign(s * down, dL) : 0.0;
}
// the raw-difference forms of the fast kind
template <int LIM>
__device__ __forceinline__ double limited_fast(double dR, double dL, q64::Range& S)
{
    const double prod = dR * dL;
    const bool use = !(prod <= 0);
    double s;
    if constexpr (LIM == LIM_MINMOD) {
        s = fabs(dR) < fabs(dL) ? dR : dL;
    } else {
        const double num = LIM == LIM_VANLEER ? prod : prod * (dR + dL);
        const double b = LIM == LIM_VANLEER ? dR + dL : dR * dR + dL * dL;
        s = q64::quo(num, q64::den(b));
        S.num_if(use, b);
    }
    return use ? s : 0.0;
}
template <int LIM>
__device__ __forceinline__ bool limited_fast_ok(double dR, double dL)
{
    return LIM == LIM_MINMOD || dR * dL <= 0 || q64::num_ok(LIM == LIM_VANLEER ? dR + dL : dR * dR + dL * dL);
}

// limited_linear_reconstruction.hpp:46-64 for NV variables of one cell along
// one dimension: values m, c, p of the cell and its neighbours, the distances
// hL, hR to them and half the cell's width (raw differences of the fast kind:
// 1, 1 and 1/2).
// One variable again, whatever its size; h_ok: both distances are in range.
template <int LIM>
static __device__ __noinline__ void face_slow(int kind, bool h_ok, double m, double c, double p, q64::Den hL, q64::Den hR,
                                              double half, double* lo, double* hi)
{
    const double aR = p - c, aL = c - m;
    double s;
    if (kind == EOS_PERFECT_GAS_FAST) {
        if (h_ok && limited_fast_ok<LIM>(aR * hR.y, aL * hL.y)) {
            return;
        }
        s = half * plain::slope(LIM, aR / hR.b, aL / hL.b, kind);
    } else {
        bool good = h_ok, pair;
        const double R = q64::quo_tiny(aR, hR, good), L = q64::quo_tiny(aL, hL, good);
        s = (LIM == LIM_VANLEER ? 2 * half : half) * limited_tiny<LIM>(R, L, pair);
        if (!(good && pair)) {
            s = half * plain::slope(LIM, aR / hR.b, aL / hL.b);
        }
    }
    *lo = c - s;
    *hi = c + s;
}
// ld(k, v): variable v of the cell (k = 1) and its neighbours (0, 2);
// ld_again(k, v) the same for the rare second look, so that a caller with the
// values in memory need not keep them in registers.
template <int NV, int LIM, class Ld, class LdAgain>
__device__ __forceinline__ void faces_ld(int kind, const Ld& ld, const LdAgain& ld_again, const q64::Den& hL,
                                         const q64::Den& hR, double half, double* lo, double* hi)
{
    const bool fast = kind == EOS_PERFECT_GAS_FAST;
    const double w = LIM == LIM_VANLEER ? 2 * half : half;
    q64::Range S;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const double c = ld(1, v);
        const double R = fast ? (ld(2, v) - c) * hR.y : q64::quo(ld(2, v) - c, hR);
        const double L = fast ? (c - ld(0, v)) * hL.y : q64::quo(c - ld(0, v), hL);
        const double s = w * (fast ? limited_fast<LIM>(R, L, S) : limited_core<LIM>(R, L, S));
        lo[v] = c - s;
        hi[v] = c + s;
    }
    const bool h_ok = q64::width_ok(hR.b) && q64::width_ok(hL.b);
    if (!(h_ok && S.ok())) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            double lt = lo[v], ht = hi[v];
            face_slow<LIM>(kind, h_ok, ld_again(0, v), ld_again(1, v), ld_again(2, v), hL, hR, half, &lt, &ht);
            lo[v] = lt;
            hi[v] = ht;
        }
    }
}
template <int NV, int LIM>
__device__ __forceinline__ void faces_den(int kind, const double* m, const double* c, const double* p, const q64::Den& hL,
                                          const q64::Den& hR, double half, double* lo, double* hi)
{
    const auto ld = [&](int k, int v) { return k == 0 ? m[v] : (k == 1 ? c[v] : p[v]); };
    faces_ld<NV, LIM>(kind, ld, ld, hL, hR, half, lo, hi);
}
template <int NV, int LIM>
__device__ __forceinline__ void faces_lim(int kind, bool uniform, const double* m, const double* c, const double* p,
                                          double dl_m, double dl, double dl_p, double* lo, double* hi)
{
    if (kind == EOS_PERFECT_GAS_FAST && uniform) {
        faces_den<NV, LIM>(kind, m, c, p, q64::Den{1.0, 1.0}, q64::Den{1.0, 1.0}, 0.5, lo, hi);
    } else {
        faces_den<NV, LIM>(kind, m, c, p, q64::den((dl_m + dl) / 2), q64::den((dl + dl_p) / 2), dl / 2, lo, hi);
    }
}
template <int NV>
__device__ __forceinline__ void faces(int kind, int lim, bool uniform, const double* m, const double* c, const double* p,
                                      double dl_m, double dl, double dl_p, double* lo, double* hi)
{
    if (lim == LIM_VANLEER) {
        faces_lim<NV, LIM_VANLEER>(kind, uniform, m, c, p, dl_m, dl, dl_p, lo, hi);
    } else if (lim == LIM_MINMOD) {
        faces_lim<NV, LIM_MINMOD>(kind, uniform, m, c, p, dl_m, dl, dl_p, lo, hi);
    } else if (lim == LIM_VANALBADA) {
        faces_lim<NV, LIM_VANALBADA>(kind, uniform, m, c, p, dl_m, dl, dl_p, lo, hi);
    } else {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            lo[v] = c[v] - ((dl / 2) * 0.0);
            hi[v] = c[v] + ((dl / 2) * 0.0);
        }
    }
}

// hydro/riemann_solver.hpp:22-134 (HLL and HLLC).  HLLC needs the flux of the
// side the star state lies on only.
template <int ND, int RS, bool TINY = false>
__device__ __forceinline__ void riemann_core(const Eos& e, const double* cL, const double* cR, int l, double* f,
                                             q64::Range& S)
{
    constexpr int NV = ND + 2;
    double pL[NV], pR[NV], evL, evR;
    q64::Den rL, rR, kL{}, kR{};
    prim_core<ND, TINY>(e, cL, pL, rL, kL, evL, S);
    prim_core<ND, TINY>(e, cR, pR, rR, kR, evR, S);
    const double PL = pL[1 + ND], PR = pR[1 + ND];
    const double aL = q64::root(q64::quo(e.gamma * PL, rL));
    const double aR = q64::root(q64::quo(e.gamma * PR, rR));
    const double uL = pL[1 + l];
    const double uR = pR[1 + l];
    const double wsL = fmin(uL - aL, uR - aR);
    const double wsR = fmax(uL + aL, uR + aR);
    // E and flux of one side's primitives (ek + e, as flux_prim)
    auto side_flux = [&](const double* p, const q64::Den& k, double* fs) {
        const double evol = e.kind == EOS_PERFECT_GAS_FAST ? p[1 + ND] * (1.0 / e.gamma_m1) : evol_core(e, p[1 + ND], k);
        double norm = 0;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            norm += p[1 + d] * p[1 + d];
        }
        const double E = __fma_rn(0.5, p[0] * norm, evol);
        const double m = p[0] * p[1 + l];
        fs[0] = m;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            fs[1 + d] = m * p[1 + d];
        }
        fs[1 + l] += p[1 + ND];
        fs[1 + ND] = p[1 + l] * (E + p[1 + ND]);
    };
    if constexpr (RS == RS_HLL) {
        double fL[NV], fR[NV];
        side_flux(pL, kL, fL);
        side_flux(pR, kR, fR);
        const double nL = fmin(wsL, 0.);
        const double nR = fmax(wsR, 0.);
        const q64::Den w = q64::den(nR - nL);
        S.den(w.b);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const double num = (nR * fL[v]) - (nL * fR[v]) + (nL * nR * (cR[v] - cL[v]));
            f[v] = num_quo<TINY>(num, w, S);
            S.num(num, num);
        }
    } else {
        const double rcL = pL[0] * (wsL - uL);
        const double rcR = pR[0] * (wsR - uR);
        const double un_num = PR - PL + (rcL * uL) - (rcR * uR);
        // rcL - rcR < 0: quo keeps a zero's sign for positive denominators
        const q64::Den du = q64::den(-(rcL - rcR));
        const double ustar = -num_quo<TINY>(un_num, du, S);
        const double pstar = 1. / 2 * (PL + PR + (rcL * (ustar - uL)) + (rcR * (ustar - uR)));
        const bool left = ustar > 0;
        const double Sw = left ? wsL : wsR;
        double cs[NV], ps[NV], fs[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            cs[v] = left ? cL[v] : cR[v];
            ps[v] = left ? pL[v] : pR[v];
        }
        side_flux(ps, q64::Den{left ? kL.b : kR.b, left ? kL.y : kR.y}, fs);
        const double un = ps[1 + l];
        const q64::Den su = q64::den(Sw - ustar);
        const double sn = Sw - un;
        const double un_s = ustar - un;
        S.den(du.b);
        S.den(su.b);
        S.add(sn);
        if (e.kind != EOS_PERFECT_GAS_FAST) {
            S.num(un_num, un_s);
        }
        double rs, Es;
        if (e.kind == EOS_PERFECT_GAS_FAST) {
            const double ratio = sn * su.y;
            rs = cs[0] * ratio;
            Es = ratio * cs[1 + ND] + un_s * su.y * (ustar * cs[0] * sn + ps[1 + ND]);
        } else {
            rs = q64::quo(cs[0] * sn, su);
            Es = (q64::quo(sn, su) * cs[1 + ND]) + (num_quo<TINY>(un_s, su, S) * ((ustar * cs[0] * sn) + ps[1 + ND]));
        }
        const double rsu = rs * ustar;
        const bool sup = wsL * wsR > 0;
        f[0] = plain::flux_hllc(fs[0], cs[0], rs, Sw);
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            f[1 + d] = rsu * ps[1 + d];
        }
        f[1 + l] = (rsu * ustar) + pstar;
        f[1 + ND] = plain::flux_hllc(fs[1 + ND], cs[1 + ND], Es, Sw);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            f[v] = sup ? fs[v] : f[v];
        }
    }
}

template <int ND, int RS, int KIND>
static __device__ __noinline__ void riemann_slow(Eos e, const double* cL, const double* cR, int l, double* f)
{
    e.kind = KIND;
    if constexpr (KIND == EOS_PERFECT_GAS) {
        q64::Range S(e.consts_ok);
        riemann_core<ND, RS, true>(e, cL, cR, l, f, S);
        if (S.dens_ok()) {
            return;
        }
    }
    plain::riemann<ND>(e, RS, cL, cR, l, f);
}
template <int ND, int RS>
__device__ __forceinline__ void riemann_rs(const Eos& e, const double* cL, const double* cR, int l, double* f)
{
    q64::Range S(e.consts_ok);
    riemann_core<ND, RS>(e, cL, cR, l, f, S);
    if (!S.ok()) {
        double lt[ND + 2], rt[ND + 2], ft[ND + 2];
#pragma unroll
        for (int v = 0; v < ND + 2; ++v) {
            lt[v] = cL[v];
            rt[v] = cR[v];
        }
        if (e.kind == EOS_PERFECT_GAS_FAST) {
            riemann_slow<ND, RS, EOS_PERFECT_GAS_FAST>(e, lt, rt, l, ft);
        } else {
            riemann_slow<ND, RS, EOS_PERFECT_GAS>(e, lt, rt, l, ft);
        }
#pragma unroll
        for (int v = 0; v < ND + 2; ++v) {
            f[v] = ft[v];
        }
    }
}

// hydro/riemann_solver.hpp:22-181.  cL/cR: conservative states; l: direction.
template <int ND>
__device__ __forceinline__ void riemann(const Eos& e, int solver, const double* cL, const double* cR, int l, double* f)
{
    if (e.kind == EOS_RAD_GAS || solver == RS_SPLITTING) {
        plain::riemann<ND>(e, solver, cL, cR, l, f);
    } else if (solver == RS_HLL) {
        riemann_rs<ND, RS_HLL>(e, cL, cR, l, f);
    } else {
        riemann_rs<ND, RS_HLLC>(e, cL, cR, l, f);
    }
}

// hydro/source_terms.hpp:16-77 (trigonometric factors precomputed on the host
// with the same libm expressions: cot_mid = cos((x1+x1p)/2)/sin((x1+x1p)/2),
// sm = sin(x1), sp = sin(x1p)).
__device__ __forceinline__ double src_grad_pres(double dtodv, double PL, double PR, double dS, double dS_p)
{
    return dtodv * (PL + PR) / 2 * (dS_p - dS);
}
__device__ __forceinline__ double src_grad_u_r(double dtodv, double rhoL, double rhoR, double uL, double uR, double dS,
                                               double dS_p)
{
    return dtodv * ((rhoL * uL * uL) + (rhoR * uR * uR)) / 2 * (dS_p - dS) / 2;
}
__device__ __forceinline__ double src_grad_u_idir_r(double dtodv, double x0, double x0_p, double rhoL, double rhoR,
                                                    double uL_r, double uR_r, double uL_o, double uR_o, double dS,
                                                    double dS_p)
{
    return dtodv * (x0_p - x0) / (x0_p + x0) * ((rhoR * uR_o * uR_r * dS_p) + (rhoL * uL_o * uL_r * dS));
}
__device__ __forceinline__ double src_grad_u_th(double dtodv, double cot_mid, double rhoL, double rhoR, double uL,
                                                double uR, double dS, double dS_p)
{
    return dtodv * ((rhoL * uL * uL) + (rhoR * uR * uR)) / 2 * cot_mid * (dS_p - dS) / 2;
}
__device__ __forceinline__ double src_grad_u_phi(double dtodv, double sm, double sp, double rhoL, double rhoR,
                                                 double uL_th, double uR_th, double uL_phi, double uR_phi, double dS,
                                                 double dS_p)
{
    return dtodv * (sp - sm) / (sp + sm) * ((rhoR * uR_phi * uR_th * dS_p) + (rhoL * uL_phi * uL_th * dS));
}

} // namespace hcl::exact
