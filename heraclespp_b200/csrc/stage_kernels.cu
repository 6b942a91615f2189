// stage_kernels.cu -- one CUDA kernel per Kokkos kernel of the reference's
// time loop, with the reference's FP64 arithmetic (this file is compiled with
// --fmad=false).  These back the stage entry points of the C ABI, which a
// maintainer wires in place of the reference's plugins; they are also the
// stage-by-stage parity path.  Iteration spaces are the reference's Ranges.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "hcl_device.cuh"
#include "physics_exact.cuh"
#include "stages.hpp"

namespace hcl {

std::atomic<int64_t> g_launches{0};

namespace {

constexpr int kThreads = 256;
// CTAs per SM that the two heaviest stage kernels are held to (120 x 100 x 70 cells,
// Van Leer and HLLC): the reconstruction 161 us at two and 260 at three, where it
// spills; the Godunov update 134 and 114 us (RadGas, waiting on branching
// divisions: 2.02 and 1.77 ms).
constexpr int kReconMinBlocks = 2;
constexpr int kGodunovMinBlocks = 3;

struct Box {
    int b[3];
    int w[3];
    int64_t count;
};

Box make_box(const GridDev& g, int ng_eff)
{
    Box bx;
    int e[3];
    cell_range(g, ng_eff, bx.b, e);
    bx.count = 1;
    for (int d = 0; d < 3; ++d) {
        bx.w[d] = e[d] - bx.b[d];
        bx.count *= bx.w[d];
    }
    return bx;
}

__device__ __forceinline__ void box_ijk(const Box& bx, int64_t idx, int& i, int& j, int& k)
{
    i = bx.b[0] + (int)(idx % bx.w[0]);
    const int64_t r = idx / bx.w[0];
    j = bx.b[1] + (int)(r % bx.w[1]);
    k = bx.b[2] + (int)(r / bx.w[1]);
}

int grid_for(int64_t count)
{
    int64_t blocks = (count + kThreads - 1) / kThreads;
    if (blocks > 148 * 16) {
        blocks = 148 * 16;
    }
    if (blocks < 1) {
        blocks = 1;
    }
    return (int)blocks;
}


// ---------------------------------------------------------------------------
// array_conversion.hpp:32-104 "conv_prim_to_cons_array"
template <int ND>
__global__ void k_prim_to_cons(GridDev g, Box bx, const double* __restrict__ rho, const double* __restrict__ u,
                               const double* __restrict__ P, double* __restrict__ rhou, double* __restrict__ E)
{
    const exact::Eos eos = exact::eos_of(g);
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < bx.count;
         idx += (int64_t)gridDim.x * blockDim.x) {
        int i, j, k;
        box_ijk(bx, idx, i, j, k);
        const int64_t c = lidx(g, i, j, k);
        double p[ND + 2], q[ND + 2];
        p[0] = rho[c];
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            p[1 + d] = u[c + g.N * d];
        }
        p[1 + ND] = P[c];
        exact::to_cons<ND>(eos, p, q);
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            rhou[c + g.N * d] = q[1 + d];
        }
        E[c] = q[1 + ND];
    }
}

// array_conversion.hpp:106-172 "conv_cons_to_prim_array"
template <int ND>
__global__ void k_cons_to_prim(GridDev g, Box bx, const double* __restrict__ rho, const double* __restrict__ rhou,
                               const double* __restrict__ E, double* __restrict__ u, double* __restrict__ P)
{
    const exact::Eos eos = exact::eos_of(g);
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < bx.count;
         idx += (int64_t)gridDim.x * blockDim.x) {
        int i, j, k;
        box_ijk(bx, idx, i, j, k);
        const int64_t c = lidx(g, i, j, k);
        double q[ND + 2], p[ND + 2];
        q[0] = rho[c];
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            q[1 + d] = rhou[c + g.N * d];
        }
        q[1 + ND] = E[c];
        exact::to_prim<ND>(eos, q, p);
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            u[c + g.N * d] = p[1 + d];
        }
        P[c] = p[1 + ND];
    }
}

// analysis/temperature.hpp:18-25 "fill_temperature_array"
__global__ void k_temperature(GridDev g, Box bx, const double* __restrict__ rho, const double* __restrict__ P,
                              double* __restrict__ T)
{
    const exact::Eos eos = exact::eos_of(g);
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < bx.count;
         idx += (int64_t)gridDim.x * blockDim.x) {
        int i, j, k;
        box_ijk(bx, idx, i, j, k);
        const int64_t c = lidx(g, i, j, k);
        T[c] = exact::temperature(eos, rho[c], P[c]);
    }
}

// limited_linear_reconstruction.hpp:46-64 "face_reconstruction":
// var_rec(c, s, idim) = rec[c + N*s + 2N*idim]
template <int ND>
__global__ void k_face_recon(GridDev g, Box bx, const double* __restrict__ var, double* __restrict__ rec)
{
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < bx.count;
         idx += (int64_t)gridDim.x * blockDim.x) {
        int i, j, k;
        box_ijk(bx, idx, i, j, k);
        const int64_t c = lidx(g, i, j, k);
        const double v = var[c];
#pragma unroll
        for (int idim = 0; idim < ND; ++idim) {
            const int ki = idim == 0, kj = idim == 1, kk = idim == 2;
            const double dl = (ki * g.dx[0][i]) + (kj * g.dx[1][j]) + (kk * g.dx[2][k]);
            const double dl_m = (ki * g.dx[0][i - ki]) + (kj * g.dx[1][j - kj]) + (kk * g.dx[2][k - kk]);
            const double dl_p = (ki * g.dx[0][i + ki]) + (kj * g.dx[1][j + kj]) + (kk * g.dx[2][k + kk]);
            const double vp = var[lidx(g, i + ki, j + kj, k + kk)];
            const double vm = var[lidx(g, i - ki, j - kj, k - kk)];
            double lo, hi;
            exact::faces<1>(EOS_PERFECT_GAS, g.limiter, false, &vm, &v, &vp, dl_m, dl, dl_p, &lo, &hi);
            rec[c + 2 * g.N * idim] = lo;
            rec[c + g.N + 2 * g.N * idim] = hi;
        }
    }
}

// The whole hydro reconstruction of one cell in one pass: limited face values
// (hydro_reconstruction.hpp:99-109), face conservatives (:111-126), the Hancock
// predictor (extrapolation_reconstruction.hpp:90-325) and the passive scalars
// (:315-339).  u_rec and P_rec receive the face velocities and pressures when
// not null; fx_rec works in place.
//
// Run as the reference's separate kernels (a reconstruction per variable, the
// conversion, the predictor) the face arrays crossed memory five times; here
// they are written once, 35 planes in and out for 3-D (41 us for 120 x 100 x 70
// at the copy rate).  The face states of all but the last dimension wait for
// the increments of the others in shared memory, where registers would spill.
template <int ND>
__global__ void __launch_bounds__(kThreads, kReconMinBlocks)
k_hydro_reconstruction(GridDev g, Box bx, double dt, const double* __restrict__ rho, const double* __restrict__ u,
                       const double* __restrict__ P, const double* __restrict__ fx, double* __restrict__ rho_rec,
                       double* __restrict__ rhou_rec, double* __restrict__ E_rec, double* __restrict__ fx_rec,
                       double* __restrict__ u_rec, double* __restrict__ P_rec)
{
    constexpr int NV = ND + 2;
    __shared__ double s_face[ND > 1 ? 2 * (ND - 1) : 1][NV][kThreads];
    const exact::Eos eos = exact::eos_of(g);
    const int64_t N = g.N;
    const int64_t S5 = 2 * N;
    const int64_t S6 = 2 * N * ND;
    const bool sph = g.geom == GEOM_SPHERICAL;
    const int tid = threadIdx.x;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < bx.count;
         idx += (int64_t)gridDim.x * blockDim.x) {
        int ijk[3];
        box_ijk(bx, idx, ijk[0], ijk[1], ijk[2]);
        const int64_t c = lidx(g, ijk[0], ijk[1], ijk[2]);
        const int64_t step[3] = {1, g.n[0], (int64_t)g.n[0] * g.n[1]};
        const double dtodv = dt / g.dv[c];
        double last[2][NV];     // faces of the last dimension
        double inc[ND][NV];     // dt/dv (F_L S_L - F_R S_R) per dimension
        double src[2][5];       // geometric terms of dimensions 0 and 1
        double mass[2][ND];
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            const double dl = g.dx[d][ijk[d]];
            const double dl_m = g.dx[d][ijk[d] - 1];
            const double dl_p = g.dx[d][ijk[d] + 1];
            double m[NV], v0[NV], p[NV], f[2][NV], U[2][NV], F[2][NV];
            const int64_t cm = c - step[d], cp = c + step[d];
            m[0] = rho[cm];
            v0[0] = rho[c];
            p[0] = rho[cp];
#pragma unroll
            for (int r = 0; r < ND; ++r) {
                m[1 + r] = u[cm + N * r];
                v0[1 + r] = u[c + N * r];
                p[1 + r] = u[cp + N * r];
            }
            m[1 + ND] = P[cm];
            v0[1 + ND] = P[c];
            p[1 + ND] = P[cp];
            exact::faces<NV>(EOS_PERFECT_GAS, g.limiter, false, m, v0, p, dl_m, dl, dl_p, f[0], f[1]);
            const double dsc = g.ds[c + N * d];
            const double dsp = g.ds[cp + N * d];
#pragma unroll
            for (int sd = 0; sd < 2; ++sd) {
                exact::to_cons_flux<ND>(eos, f[sd], d, U[sd], F[sd]);
                mass[sd][d] = F[sd][0];
                const int64_t o = c + N * sd + S5 * d;
                if (u_rec) {
#pragma unroll
                    for (int r = 0; r < ND; ++r) {
                        u_rec[o + S6 * r] = f[sd][1 + r];
                    }
                }
                if (P_rec) {
                    P_rec[o] = f[sd][1 + ND];
                }
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    if (d == ND - 1) {
                        last[sd][v] = U[sd][v];
                    } else {
                        s_face[2 * d + sd][v][tid] = U[sd][v];
                    }
                }
            }
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                inc[d][v] = dtodv * ((F[0][v] * dsc) - (F[1][v] * dsp));
            }
            if (sph) { // :145-303
                const double *pL = f[0], *pR = f[1];
                if (d == 0) {
                    src[0][0] = exact::src_grad_pres(dtodv, pL[1 + ND], pR[1 + ND], dsc, dsp);
                    if constexpr (ND >= 2) {
                        src[0][1] = exact::src_grad_u_r(dtodv, pL[0], pR[0], pL[2], pR[2], dsc, dsp);
                        src[0][2] = exact::src_grad_u_idir_r(dtodv, g.x[0][ijk[0]], g.x[0][ijk[0] + 1], pL[0], pR[0],
                                                             pL[1], pR[1], pL[2], pR[2], dsc, dsp);
                    }
                    if constexpr (ND == 3) {
                        src[0][3] = exact::src_grad_u_r(dtodv, pL[0], pR[0], pL[3], pR[3], dsc, dsp);
                        src[0][4] = exact::src_grad_u_idir_r(dtodv, g.x[0][ijk[0]], g.x[0][ijk[0] + 1], pL[0], pR[0],
                                                             pL[1], pR[1], pL[3], pR[3], dsc, dsp);
                    }
                }
                if (d == 1) {
                    src[1][0] = exact::src_grad_pres(dtodv, pL[1 + ND], pR[1 + ND], dsc, dsp);
                    if constexpr (ND == 3) {
                        src[1][1] = exact::src_grad_u_th(dtodv, g.cot_mid1[ijk[1]], pL[0], pR[0], pL[3], pR[3], dsc, dsp);
                        src[1][2] = exact::src_grad_u_phi(dtodv, g.sin1[ijk[1]], g.sin1[ijk[1] + 1], pL[0], pR[0], pL[2],
                                                          pR[2], pL[3], pR[3], dsc, dsp);
                    }
                }
            }
        }
        double rho_old[2][ND], rho_new[2][ND];
#pragma unroll
        for (int ip = 0; ip < ND; ++ip) {
#pragma unroll
            for (int sd = 0; sd < 2; ++sd) {
                double U[NV];
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    U[v] = ip == ND - 1 ? last[sd][v] : s_face[2 * ip + sd][v][tid];
                }
                const double old0 = U[0];
                double mom[ND];
#pragma unroll
                for (int r = 0; r < ND; ++r) {
                    mom[r] = U[1 + r];
                }
#pragma unroll
                for (int d = 0; d < ND; ++d) {
#pragma unroll
                    for (int v = 0; v < NV; ++v) {
                        U[v] += inc[d][v];
                    }
                    if (sph && d == 0) {
                        U[1] += src[0][0];
                        if constexpr (ND >= 2) {
                            U[1] += src[0][1];
                            U[2] -= src[0][2];
                        }
                        if constexpr (ND == 3) {
                            U[1] += src[0][3];
                            U[3] -= src[0][4];
                        }
                    }
                    if constexpr (ND >= 2) {
                        if (sph && d == 1) {
                            U[2] += src[1][0];
                            if constexpr (ND == 3) {
                                U[2] += src[1][1];
                                U[3] -= src[1][2];
                            }
                        }
                    }
                    const double gd = gravity_at(g, ijk[0], d); // :306-312
                    U[1 + d] += dt * gd * old0;
                    U[1 + ND] += dt * gd * mom[d];
                }
                rho_old[sd][ip] = old0;
                rho_new[sd][ip] = U[0];
                const int64_t o = c + N * sd + S5 * ip;
                rho_rec[o] = U[0];
#pragma unroll
                for (int r = 0; r < ND; ++r) {
                    rhou_rec[o + S6 * r] = U[1 + r];
                }
                E_rec[o] = U[1 + ND];
            }
        }
        for (int f = 0; f < g.nfx; ++f) {
            const double* x = fx + N * f;
            double xf[2][ND];
#pragma unroll
            for (int d = 0; d < ND; ++d) {
                const double m = x[c - step[d]], v0 = x[c], p = x[c + step[d]];
                exact::faces<1>(EOS_PERFECT_GAS, g.limiter, false, &m, &v0, &p, g.dx[d][ijk[d] - 1], g.dx[d][ijk[d]],
                                g.dx[d][ijk[d] + 1], &xf[0][d], &xf[1][d]);
            }
#pragma unroll
            for (int ip = 0; ip < ND; ++ip) {
#pragma unroll
                for (int sd = 0; sd < 2; ++sd) {
                    double v = xf[sd][ip] * rho_old[sd][ip];
#pragma unroll
                    for (int d = 0; d < ND; ++d) {
                        const double dsc = g.ds[c + N * d];
                        const double dsp = g.ds[c + step[d] + N * d];
                        v += dtodv * (((xf[0][d] * mass[0][d]) * dsc) - ((xf[1][d] * mass[1][d]) * dsp));
                    }
                    fx_rec[c + N * sd + S5 * ip + S6 * f] = v / rho_new[sd][ip];
                }
            }
        }
    }
}

// godunov_scheme.hpp:110-292 "Riemann_based_Godunov_scheme" on tiles: each
// face's Riemann problem is solved once (the reference solves it from both
// sides), its flux kept in shared memory, then every cell of the tile updates.
// 32 x 4 x 2 cells in 3-D: 968 faces instead of 1536 solves.  A warp takes rows
// of 32 faces of one dimension; the tile's last x-faces form one more row.
template <int ND>
struct GodTile {
    static constexpr int T[3] = {ND == 1 ? kThreads : 32, ND == 1 ? 1 : (ND == 2 ? 8 : 4), ND == 3 ? 2 : 1};
    static constexpr int NF(int d)
    {
        return (T[0] + (d == 0)) * (T[1] + (d == 1)) * (T[2] + (d == 2));
    }
    static constexpr int off(int d)
    {
        return d == 0 ? 0 : (d == 1 ? NF(0) : NF(0) + NF(1));
    }
    static constexpr int total = NF(0) + (ND > 1 ? NF(1) : 0) + (ND > 2 ? NF(2) : 0);
};

template <int ND>
__global__ void __launch_bounds__(kThreads, kGodunovMinBlocks) k_godunov(GridDev g, Box bx, double dt, const double* __restrict__ rho, const double* __restrict__ rhou,
                          const double* __restrict__ E, const double* __restrict__ fx,
                          const double* __restrict__ rho_rec, const double* __restrict__ rhou_rec,
                          const double* __restrict__ E_rec, const double* __restrict__ fx_rec,
                          double* __restrict__ rho_new, double* __restrict__ rhou_new, double* __restrict__ E_new,
                          double* __restrict__ fx_new)
{
    using T = GodTile<ND>;
    constexpr int NV = ND + 2;
    constexpr int T0 = T::T[0], T1 = T::T[1], T2 = T::T[2];
    __shared__ double s_flux[NV][T::total];
    const exact::Eos eos = exact::eos_of(g);
    const int64_t N = g.N;
    const int64_t S5 = 2 * N;
    const int64_t S6 = 2 * N * ND;
    const bool sph = g.geom == GEOM_SPHERICAL;
    const int64_t step[3] = {1, g.n[0], (int64_t)g.n[0] * g.n[1]};
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int nt0 = (bx.w[0] + T0 - 1) / T0;
    const int nt1 = (bx.w[1] + T1 - 1) / T1;
    const int org[3] = {bx.b[0] + (int)(blockIdx.x % nt0) * T0, bx.b[1] + (int)(blockIdx.x / nt0 % nt1) * T1,
                        bx.b[2] + (int)(blockIdx.x / nt0 / nt1) * T2};
    const int end[3] = {bx.b[0] + bx.w[0], bx.b[1] + bx.w[1], bx.b[2] + bx.w[2]};

    // face f = (a0, a1, a2) of dimension d: between the cells at org + a - 1_d
    // and org + a
    auto solve = [&](auto dc, int a0, int a1, int a2) {
        constexpr int d = decltype(dc)::value;
        const int i = org[0] + a0, j = org[1] + a1, k = org[2] + a2;
        if (i >= end[0] + (d == 0) || j >= end[1] + (d == 1) || k >= end[2] + (d == 2)) {
            return;
        }
        const int64_t c = lidx(g, i, j, k);
        const int64_t oL = c - step[d] + N + S5 * d; // right state of the left cell
        const int64_t oR = c + S5 * d;
        double cL[NV], cR[NV], F[NV];
        cL[0] = rho_rec[oL];
        cR[0] = rho_rec[oR];
#pragma unroll
        for (int r = 0; r < ND; ++r) {
            cL[1 + r] = rhou_rec[oL + S6 * r];
            cR[1 + r] = rhou_rec[oR + S6 * r];
        }
        cL[1 + ND] = E_rec[oL];
        cR[1 + ND] = E_rec[oR];
        exact::riemann<ND>(eos, g.riemann, cL, cR, d, F);
        const int f = T::off(d) + a0 + (T0 + (d == 0)) * (a1 + (T1 + (d == 1)) * a2);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            s_flux[v][f] = F[v];
        }
    };
    constexpr int B0 = T0 / 32;          // row blocks along x
    constexpr int R0 = B0 * T1 * T2;     // rows of x-faces
    constexpr int RX = (T1 * T2 + 31) / 32; // the last x-faces
    constexpr int R1 = ND > 1 ? B0 * (T1 + 1) * T2 : 0;
    constexpr int R2 = ND > 2 ? B0 * T1 * (T2 + 1) : 0;
#pragma unroll 1
    for (int t = tid >> 5; t < R0 + RX + R1 + R2; t += kThreads / 32) {
        if (t < R0) {
            const int q = t / B0;
            solve(std::integral_constant<int, 0>{}, (t % B0) * 32 + lane, q % T1, q / T1);
        } else if (t < R0 + RX) {
            const int q = (t - R0) * 32 + lane;
            if (q < T1 * T2) {
                solve(std::integral_constant<int, 0>{}, T0, q % T1, q / T1);
            }
        } else if (t < R0 + RX + R1) {
            if constexpr (ND > 1) {
                const int r = t - R0 - RX, q = r / B0;
                solve(std::integral_constant<int, 1>{}, (r % B0) * 32 + lane, q % (T1 + 1), q / (T1 + 1));
            }
        } else {
            if constexpr (ND > 2) {
                const int r = t - R0 - RX - R1, q = r / B0;
                solve(std::integral_constant<int, 2>{}, (r % B0) * 32 + lane, q % T1, q / T1);
            }
        }
    }
    __syncthreads();

    const int x[3] = {tid % T0, tid / T0 % T1, tid / T0 / T1};
    const int i = org[0] + x[0], j = org[1] + x[1], k = org[2] + x[2];
    if (i >= end[0] || j >= end[1] || k >= end[2]) {
        return;
    }
    const int64_t c = lidx(g, i, j, k);
    const double r_old = rho[c];
    double rn = r_old;
    double En = E[c];
    double mo[ND], mn[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        mo[d] = mn[d] = rhou[c + N * d];
    }
    for (int f = 0; f < g.nfx; ++f) {
        fx_new[c + N * f] = fx[c + N * f] * r_old;
    }
    const double dtodv = dt / g.dv[c];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        const int64_t cm = c - step[d], cp = c + step[d];
        const int fL = T::off(d) + x[0] + (T0 + (d == 0)) * (x[1] + (T1 + (d == 1)) * x[2]);
        const int fR = fL + (d == 0 ? 1 : (d == 1 ? T0 : T0 * T1));
        double FL[NV], FR[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            FL[v] = s_flux[v][fL];
            FR[v] = s_flux[v][fR];
        }
        const double dsc = g.ds[c + N * d];
        const double dsp = g.ds[cp + N * d];
        rn += dtodv * ((FL[0] * dsc) - (FR[0] * dsp));
#pragma unroll
        for (int r = 0; r < ND; ++r) {
            mn[r] += dtodv * ((FL[1 + r] * dsc) - (FR[1 + r] * dsp));
        }
        En += dtodv * ((FL[1 + ND] * dsc) - (FR[1 + ND] * dsp));
        if (sph && d < 2) {
            // :165-256, from the cell's own face states
            double vL[NV], vR[NV], pl[NV], pr[NV];
            const int64_t o = c + S5 * d;
            vL[0] = rho_rec[o];
            vR[0] = rho_rec[o + N];
#pragma unroll
            for (int r = 0; r < ND; ++r) {
                vL[1 + r] = rhou_rec[o + S6 * r];
                vR[1 + r] = rhou_rec[o + N + S6 * r];
            }
            vL[1 + ND] = E_rec[o];
            vR[1 + ND] = E_rec[o + N];
            exact::to_prim<ND>(eos, vL, pl);
            exact::to_prim<ND>(eos, vR, pr);
            if (d == 0) {
                mn[0] += exact::src_grad_pres(dtodv, pl[1 + ND], pr[1 + ND], dsc, dsp);
                if constexpr (ND >= 2) {
                    mn[0] += exact::src_grad_u_r(dtodv, pl[0], pr[0], pl[2], pr[2], dsc, dsp);
                    mn[1] -= exact::src_grad_u_idir_r(dtodv, g.x[0][i], g.x[0][i + 1], pl[0], pr[0], pl[1], pr[1],
                                                      pl[2], pr[2], dsc, dsp);
                }
                if constexpr (ND == 3) {
                    mn[0] += exact::src_grad_u_r(dtodv, pl[0], pr[0], pl[3], pr[3], dsc, dsp);
                    mn[2] -= exact::src_grad_u_idir_r(dtodv, g.x[0][i], g.x[0][i + 1], pl[0], pr[0], pl[1], pr[1],
                                                      pl[3], pr[3], dsc, dsp);
                }
            }
            if constexpr (ND >= 2) {
                if (d == 1) {
                    mn[1] += exact::src_grad_pres(dtodv, pl[1 + ND], pr[1 + ND], dsc, dsp);
                    if constexpr (ND == 3) {
                        mn[1] += exact::src_grad_u_th(dtodv, g.cot_mid1[j], pl[0], pr[0], pl[3], pr[3], dsc, dsp);
                        mn[2] -= exact::src_grad_u_phi(dtodv, g.sin1[j], g.sin1[j + 1], pl[0], pr[0], pl[2], pr[2],
                                                       pl[3], pr[3], dsc, dsp);
                    }
                }
            }
        }
        // gravity :258-260
        const double gd = gravity_at(g, i, d);
        mn[d] += dt * gd * r_old;
        En += dt * gd * mo[d];
        // passive scalars :262-290
        for (int f = 0; f < g.nfx; ++f) {
            const int64_t off = S6 * f + S5 * d;
            const double ffL = fx_rec[(FL[0] < 0 ? c : cm + N) + off] * FL[0];
            const double ffR = fx_rec[(FR[0] < 0 ? cp : c + N) + off] * FR[0];
            fx_new[c + N * f] += dtodv * ((ffL * dsc) - (ffR * dsp));
        }
    }
    rho_new[c] = rn;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        rhou_new[c + N * d] = mn[d];
    }
    E_new[c] = En;
}

// pressure_fix.hpp:19-172: where the old internal energy is below eps times
// the kinetic energy, E_new is rebuilt from a blend of the Godunov increment
// and a pressure-work estimate from the face velocities (the reference's loop
// order, including the overwrite of E_new inside the inner loop)
template <int ND>
__global__ void k_pressure_fix(GridDev g, Box bx, double dt, double eps, const double* __restrict__ rho,
                               const double* __restrict__ rhou, const double* __restrict__ E,
                               const double* __restrict__ rho_rec, const double* __restrict__ rhou_rec,
                               const double* __restrict__ E_rec, const double* __restrict__ rho_new,
                               const double* __restrict__ rhou_new, double* __restrict__ E_new)
{
    const exact::Eos eos = exact::eos_of(g);
    const int64_t N = g.N;
    const int64_t S5 = 2 * N;
    const int64_t S6 = 2 * N * ND;
    const double eps2 = eps / 10;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < bx.count;
         idx += (int64_t)gridDim.x * blockDim.x) {
        int i, j, k;
        box_ijk(bx, idx, i, j, k);
        const int64_t c = lidx(g, i, j, k);
        double cons[ND + 2], cons_new[ND + 2], prim[ND + 2];
        cons[0] = rho[c];
        cons_new[0] = rho_new[c];
#pragma unroll
        for (int r = 0; r < ND; ++r) {
            cons[1 + r] = rhou[c + N * r];
            cons_new[1 + r] = rhou_new[c + N * r];
        }
        cons[1 + ND] = E[c];
        cons_new[1 + ND] = E_new[c];
        exact::to_prim<ND>(eos, cons, prim);
        const double ekin = exact::ek_cons<ND>(cons);
        const double evol = E[c] - ekin;
        const double evol_new = E_new[c] - exact::ek_cons<ND>(cons_new);
        const double de_god = evol_new - evol;
        if (!(evol < eps * ekin)) {
            continue;
        }
        double En = E[c];
        double divU = 0;
        double divUE = 0;
        double einL = 0;
        double einR = 0;
        double alpha = (evol * evol) / (ekin * ekin * eps * eps);
        if (evol < eps2 * ekin) {
            alpha = 0;
        }
        for (int idim = 0; idim < ND; ++idim) {
            const int64_t cm = lidx(g, i - (idim == 0), j - (idim == 1), k - (idim == 2));
            const int64_t cp = lidx(g, i + (idim == 0), j + (idim == 1), k + (idim == 2));
            for (int ipos = 0; ipos < ND; ++ipos) {
                double vL[ND + 2], vR[ND + 2], mR[ND + 2], pL[ND + 2], cons_p[ND + 2], cons_m[ND + 2];
                double primL[ND + 2], primR[ND + 2], prim_mR[ND + 2], prim_pL[ND + 2];
                vL[0] = rho_rec[c + S5 * idim];
                vR[0] = rho_rec[c + N + S5 * idim];
                mR[0] = rho_rec[cm + N + S5 * idim];
                pL[0] = rho_rec[cp + S5 * idim];
                cons_p[0] = rho[cp];
                cons_m[0] = rho[cm];
#pragma unroll
                for (int r = 0; r < ND; ++r) {
                    vL[1 + r] = rhou_rec[c + S5 * idim + S6 * r];
                    vR[1 + r] = rhou_rec[c + N + S5 * idim + S6 * r];
                    mR[1 + r] = rhou_rec[cm + N + S5 * idim + S6 * r];
                    pL[1 + r] = rhou_rec[cp + S5 * idim + S6 * r];
                    cons_p[1 + r] = rhou[cp + N * r];
                    cons_m[1 + r] = rhou[cm + N * r];
                }
                vL[1 + ND] = E_rec[c + S5 * idim];
                vR[1 + ND] = E_rec[c + N + S5 * idim];
                mR[1 + ND] = E_rec[cm + N + S5 * idim];
                pL[1 + ND] = E_rec[cp + S5 * idim];
                cons_p[1 + ND] = E[cp];
                cons_m[1 + ND] = E[cm];
                exact::to_prim<ND>(eos, vL, primL);
                exact::to_prim<ND>(eos, vR, primR);
                exact::to_prim<ND>(eos, mR, prim_mR);
                exact::to_prim<ND>(eos, pL, prim_pL);
                const double us = (prim_mR[1 + ipos] + primL[1 + ipos]) / 2;
                const double us_p = (primR[1 + ipos] + prim_pL[1 + ipos]) / 2;
                divU += ((us_p * g.ds[cp + N * ipos]) - (us * g.ds[c + N * ipos])) / g.dv[c];
                if (us_p > 0) {
                    einR = E[c] - exact::ek_cons<ND>(cons);
                } else {
                    einR = E[cp] - exact::ek_cons<ND>(cons_p);
                }
                if (us < 0) {
                    einL = E[c] - exact::ek_cons<ND>(cons);
                } else {
                    einL = E[cm] - exact::ek_cons<ND>(cons_m);
                }
                divUE += ((us_p * einR * g.ds[cp + N * ipos]) - (us * einL * g.ds[c + N * ipos])) / g.dv[c];
                const double de_pf = dt * ((-prim[1 + ND] * divU) - divUE);
                double sum = 0;
#pragma unroll
                for (int idr = 0; idr < ND; ++idr) {
                    sum += cons[1 + idr] * cons[1 + idr] / cons[0];
                }
                const double de_tot = (alpha * de_god) + ((1 - alpha) * de_pf);
                En = evol + de_tot + (1. / 2 * sum);
            }
        }
        E_new[c] = En;
    }
}

// godunov_scheme.hpp:294-301 "passive_scalar_Godunov"
__global__ void k_passive_godunov(GridDev g, Box bx, const double* __restrict__ rho_new, double* __restrict__ fx_new)
{
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < bx.count;
         idx += (int64_t)gridDim.x * blockDim.x) {
        int i, j, k;
        box_ijk(bx, idx, i, j, k);
        const int64_t c = lidx(g, i, j, k);
        for (int f = 0; f < g.nfx; ++f) {
            const double v = fx_new[c + g.N * f] / rho_new[c];
            fx_new[c + g.N * f] = v < 0. ? 0. : (v > 1. ? 1. : v);
        }
    }
}

// boundary_distribute.hpp:42-76 on one rank, as a gather (see bc_source)
template <int ND>
__global__ void k_fill_ghosts(GridDev g, double* __restrict__ rho, double* __restrict__ rhou, double* __restrict__ E,
                              double* __restrict__ fx)
{
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < g.N; c += (int64_t)gridDim.x * blockDim.x) {
        int idx[3];
        idx[0] = (int)(c % g.n[0]);
        const int64_t r = c / g.n[0];
        idx[1] = (int)(r % g.n[1]);
        idx[2] = (int)(r / g.n[1]);
        int src[3] = {idx[0], idx[1], idx[2]};
        int flip[3] = {0, 0, 0};
        bool ghost = false;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            src[d] = bc_source(idx[d], g.n[d], g.ng, g.bc[2 * d], g.bc[2 * d + 1], &flip[d]);
            ghost |= src[d] != idx[d];
        }
        if (!ghost) {
            continue;
        }
        const int64_t s = lidx(g, src[0], src[1], src[2]);
        rho[c] = rho[s];
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            const double v = rhou[s + g.N * d];
            rhou[c + g.N * d] = flip[d] ? -v : v;
        }
        E[c] = E[s];
        for (int f = 0; f < g.nfx; ++f) {
            fx[c + g.N * f] = fx[s + g.N * f];
        }
    }
}

__device__ __forceinline__ double warp_max(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    }
    return v;
}

// time_step.hpp:55-77 "time_step" (Max reducer): per-cell sum_d (|u_d|+c)/dx_geom_d
template <int ND>
__global__ void k_time_step(GridDev g, Box bx, const double* __restrict__ rho, const double* __restrict__ u,
                            const double* __restrict__ P, unsigned long long* inv_bits)
{
    const exact::Eos eos = exact::eos_of(g);
    double local = 0;
    bool has_nan = false;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < bx.count;
         idx += (int64_t)gridDim.x * blockDim.x) {
        int i, j, k;
        box_ijk(bx, idx, i, j, k);
        const int64_t c = lidx(g, i, j, k);
        const double sound = exact::sound(eos, rho[c], P[c]);
        double dxg[3] = {g.dx[0][i], g.dx[1][j], g.dx[2][k]};
        if (g.geom == GEOM_SPHERICAL) {
            if (ND == 2) {
                dxg[1] *= g.xc[0][i];
            }
            if (ND == 3) {
                dxg[1] *= g.xc[0][i];
                dxg[2] *= g.xc[0][i] * g.sin_xc1[j];
            }
        }
        double cell = 0;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            cell += (fabs(u[c + g.N * d]) + sound) / dxg[d];
        }
        has_nan |= isnan(cell);
        local = local > cell ? local : cell;
    }
    local = warp_max(local);
    __shared__ double red[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) {
        red[w] = local;
    }
    __syncthreads();
    if (w == 0) {
        local = lane < (int)(blockDim.x >> 5) ? red[lane] : 0.0;
        local = warp_max(local);
        if (lane == 0) {
            atomicMax(inv_bits, dbl_bits(local));
        }
    }
    if (has_nan) {
        atomicMax(inv_bits, 0x7ff8000000000000ull);
    }
}

// ordered key for doubles of any sign: monotone under unsigned compare
__device__ __forceinline__ unsigned long long min_key(double v)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

// internal_energy.cpp:25-42 "min_internal_energy" over no_ghosts
template <int ND>
__global__ void k_min_evol(GridDev g, Box bx, const double* __restrict__ rho, const double* __restrict__ rhou,
                           const double* __restrict__ E, unsigned long long* key, int* nan_flag)
{
    unsigned long long local = ~0ull;
    bool has_nan = false;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < bx.count;
         idx += (int64_t)gridDim.x * blockDim.x) {
        int i, j, k;
        box_ijk(bx, idx, i, j, k);
        const int64_t c = lidx(g, i, j, k);
        double q[ND + 2];
        q[0] = rho[c];
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            q[1 + d] = rhou[c + g.N * d];
        }
        q[1 + ND] = E[c];
        const double ev = q[1 + ND] - exact::ek_cons<ND>(q);
        if (isnan(ev)) {
            has_nan = true;
        } else {
            const unsigned long long kk = min_key(ev);
            local = kk < local ? kk : local;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, local, o);
        local = other < local ? other : local;
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(key, local);
    }
    if (has_nan) {
        atomicOr(nan_flag, 1);
    }
}

// Compensated (TwoSum) partial sums of var*dv, one pair per block.
__device__ __forceinline__ void two_sum_acc(double& s, double& e, double v)
{
    const double t = s + v;
    const double bp = t - s;
    e += (s - (t - bp)) + (v - bp);
    s = t;
}

constexpr int kRedBlocks = 296;

__global__ void k_integrate_partial(GridDev g, Box bx, const double* __restrict__ var, double* partials)
{
    double s = 0, e = 0;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < bx.count;
         idx += (int64_t)gridDim.x * blockDim.x) {
        int i, j, k;
        box_ijk(bx, idx, i, j, k);
        const int64_t c = lidx(g, i, j, k);
        two_sum_acc(s, e, var[c] * g.dv[c]);
    }
    __shared__ double ss[kThreads], se[kThreads];
    ss[threadIdx.x] = s;
    se[threadIdx.x] = e;
    __syncthreads();
    if (threadIdx.x == 0) {
        double S = 0, Ecomp = 0;
        for (int t = 0; t < (int)blockDim.x; ++t) {
            two_sum_acc(S, Ecomp, ss[t]);
            Ecomp += se[t];
        }
        partials[2 * blockIdx.x] = S;
        partials[2 * blockIdx.x + 1] = Ecomp;
    }
}

__global__ void k_integrate_final(const double* partials, int nblocks, double* out)
{
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        double S = 0, Ecomp = 0;
        for (int b = 0; b < nblocks; ++b) {
            two_sum_acc(S, Ecomp, partials[2 * b]);
            Ecomp += partials[2 * b + 1];
        }
        out[0] = S + Ecomp;
        out[1] = Ecomp;
    }
}

template <class F>
void dispatch_nd(int nd, F&& f)
{
    if (nd == 1) {
        f(std::integral_constant<int, 1>{});
    } else if (nd == 2) {
        f(std::integral_constant<int, 2>{});
    } else {
        f(std::integral_constant<int, 3>{});
    }
}

// InternalMassGravity (gravity.cpp:59-128): the shell means of rho, then the
// enclosed mass and the radial table g = -G M / xc^2.  rho has rows of `pitch`
// doubles (n0 for the reference layout); shell: nx0 + ng doubles of scratch;
// g_r: n0 doubles (the handle's radial table).
//
// A shell's mean is a sum over (j, k) in a fixed order (j outer, k inner), one
// dependent addition per cell, so its floor is the addition's latency: 3200
// cells of a 96 x 64 x 50 grid, ~15 us.  A CTA sums 32 shells with one warp
// while its other warps bring in the products rho dv of the next chunks through
// registers and shared memory, two chunks ahead of the sum.  One thread per
// shell that loads for itself waits out each load: 954 us; loads not issued
// ahead: 169 us; so: 57 us.  The shells' volumes do not change and come from the host
// (g.shell_dv).
constexpr int kShellWarps = 16;
constexpr int kShellChunk = 96; // 2 buffers x 96 x 32 doubles = 48 KB
__global__ void __launch_bounds__(32 * kShellWarps) k_shell_means(GridDev g, const double* __restrict__ rho, int pitch,
                                                                  double* __restrict__ shell)
{
    constexpr int kLoaders = kShellWarps - 1;
    constexpr int kPer = (kShellChunk + kLoaders - 1) / kLoaders; // rows of a loader per chunk
    __shared__ double buf[2][kShellChunk][32];
    const int lane = threadIdx.x & 31;
    const int w = threadIdx.x >> 5;
    const int nsh = g.nx[0] + g.ng;
    const int sh = blockIdx.x * 32 + lane;
    const int i = min(sh, nsh - 1) + g.ng;
    const int g1 = g.ndim >= 2 ? g.ng : 0;
    const int g2 = g.ndim >= 3 ? g.ng : 0;
    const unsigned nk = g.nx[2];
    const unsigned count = (unsigned)g.nx[1] * nk;
    double r[kPer], v[kPer];
    auto load = [&](unsigned c0) {
#pragma unroll
        for (int m = 0; m < kPer; ++m) {
            const unsigned q = (w - 1) + kLoaders * m;
            const unsigned c = c0 + q;
            r[m] = v[m] = 0.0;
            if (q < kShellChunk && c < count) {
                const int j = (int)(c / nk) + g1;
                const int k = (int)(c % nk) + g2;
                r[m] = rho[((int64_t)k * g.n[1] + j) * pitch + i];
                v[m] = g.dv[lidx(g, i, j, k)];
            }
        }
    };
    auto store = [&](int b) {
#pragma unroll
        for (int m = 0; m < kPer; ++m) {
            const int q = (w - 1) + kLoaders * m;
            if (q < kShellChunk) {
                buf[b][q][lane] = r[m] * v[m];
            }
        }
    };
    if (w > 0) {
        load(0);
        store(0);
        load(kShellChunk);
    }
    __syncthreads();
    double sm = 0;
    int b = 0;
    for (unsigned c0 = 0; c0 < count; c0 += kShellChunk, b ^= 1) {
        if (w > 0) {
            store(b ^ 1);
            load(c0 + 2 * kShellChunk);
        } else if (count - c0 >= kShellChunk) {
#pragma unroll 16
            for (int q = 0; q < kShellChunk; ++q) {
                sm += buf[b][q][lane];
            }
        } else {
            for (int q = 0; q < (int)(count - c0); ++q) {
                sm += buf[b][q][lane];
            }
        }
        __syncthreads();
    }
    if (w == 0 && sh < nsh) {
        shell[sh] = sm / g.shell_dv[sh];
    }
}

// The enclosed mass runs outwards from the central mass in order; its terms
// are formed in parallel, a chunk of radii at a time.
constexpr int kMassThreads = 256;
__global__ void __launch_bounds__(kMassThreads) k_internal_mass_gravity(GridDev g, double central_mass,
                                                                        const double* __restrict__ shell,
                                                                        double* __restrict__ g_r)
{
    __shared__ double term[kMassThreads];
    const int ng = g.ng;
    const double* x0 = g.x[0];
    const double* xc = g.xc[0];
    const double vol_s3 = 4 * kPi / 3;
    double partial = 0;
    for (int c0 = 0; c0 < g.n[0]; c0 += kMassThreads) {
        const int i = c0 + threadIdx.x;
        if (i < ng) {
            term[threadIdx.x] = central_mass;
        } else if (i < g.n[0]) {
            const int off = i - ng;
            const double x3 = x0[i] * x0[i] * x0[i];
            const double up = vol_s3 * ((xc[i] * xc[i] * xc[i]) - x3) * shell[off];
            term[threadIdx.x] =
                i == ng ? central_mass + up
                        : (vol_s3 * (x3 - (xc[i - 1] * xc[i - 1] * xc[i - 1])) * shell[off - 1]) + up;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            const int m = min(kMassThreads, g.n[0] - c0);
            for (int r = c0 < ng ? ng - c0 : 0; r < m; ++r) {
                partial += term[r];
                term[r] = partial;
            }
        }
        __syncthreads();
        if (i < g.n[0]) {
            g_r[i] = -kG * term[threadIdx.x] / (xc[i] * xc[i]);
        }
        __syncthreads();
    }
}

} // namespace

namespace stage {

void conv_prim_to_cons(const GridDev& g, int ng_eff, const double* rho, const double* u, const double* P,
                       double* rhou, double* E, cudaStream_t s)
{
    const Box bx = make_box(g, ng_eff);
    dispatch_nd(g.ndim, [&](auto nd) {
        k_prim_to_cons<decltype(nd)::value><<<grid_for(bx.count), kThreads, 0, s>>>(g, bx, rho, u, P, rhou, E);
    });
    ++g_launches;
}

void conv_cons_to_prim(const GridDev& g, int ng_eff, const double* rho, const double* rhou, const double* E,
                       double* u, double* P, cudaStream_t s)
{
    const Box bx = make_box(g, ng_eff);
    dispatch_nd(g.ndim, [&](auto nd) {
        k_cons_to_prim<decltype(nd)::value><<<grid_for(bx.count), kThreads, 0, s>>>(g, bx, rho, rhou, E, u, P);
    });
    ++g_launches;
}

void temperature(const GridDev& g, int ng_eff, const double* rho, const double* P, double* T, cudaStream_t s)
{
    const Box bx = make_box(g, ng_eff);
    k_temperature<<<grid_for(bx.count), kThreads, 0, s>>>(g, bx, rho, P, T);
    ++g_launches;
}

void face_reconstruction(const GridDev& g, int ng_eff, const double* var, double* var_rec, cudaStream_t s)
{
    const Box bx = make_box(g, ng_eff);
    dispatch_nd(g.ndim, [&](auto nd) {
        k_face_recon<decltype(nd)::value><<<grid_for(bx.count), kThreads, 0, s>>>(g, bx, var, var_rec);
    });
    ++g_launches;
}

void hydro_reconstruction(const GridDev& g, int ng_eff, double dt, const double* rho, const double* u,
                          const double* P, const double* fx, double* rho_rec, double* rhou_rec, double* E_rec,
                          double* fx_rec, double* u_rec, double* P_rec, cudaStream_t s)
{
    const Box bx = make_box(g, ng_eff);
    dispatch_nd(g.ndim, [&](auto ndc) {
        constexpr int ND = decltype(ndc)::value;
        k_hydro_reconstruction<ND><<<grid_for(bx.count), kThreads, 0, s>>>(g, bx, dt, rho, u, P, fx, rho_rec, rhou_rec,
                                                                           E_rec, fx_rec, u_rec, P_rec);
    });
    ++g_launches;
}

void godunov(const GridDev& g, int ng_eff, double dt, const double* rho, const double* rhou, const double* E,
             const double* fx, const double* rho_rec, const double* rhou_rec, const double* E_rec,
             const double* fx_rec, double* rho_new, double* rhou_new, double* E_new, double* fx_new,
             cudaStream_t s)
{
    const Box bx = make_box(g, ng_eff);
    dispatch_nd(g.ndim, [&](auto ndc) {
        constexpr int ND = decltype(ndc)::value;
        using T = GodTile<ND>;
        const int64_t blocks = (int64_t)((bx.w[0] + T::T[0] - 1) / T::T[0]) * ((bx.w[1] + T::T[1] - 1) / T::T[1]) *
                               ((bx.w[2] + T::T[2] - 1) / T::T[2]);
        k_godunov<ND><<<(unsigned)blocks, kThreads, 0, s>>>(g, bx, dt, rho, rhou, E, fx, rho_rec, rhou_rec, E_rec,
                                                              fx_rec, rho_new, rhou_new, E_new, fx_new);
    });
    ++g_launches;
    if (g.nfx > 0) {
        k_passive_godunov<<<grid_for(bx.count), kThreads, 0, s>>>(g, bx, rho_new, fx_new);
        ++g_launches;
    }
}

void pressure_fix(const GridDev& g, double dt, double eps, const double* rho, const double* rhou, const double* E,
                  const double* rho_rec, const double* rhou_rec, const double* E_rec, const double* rho_new,
                  const double* rhou_new, double* E_new, cudaStream_t s)
{
    const Box bx = make_box(g, 0);
    dispatch_nd(g.ndim, [&](auto ndc) {
        constexpr int ND = decltype(ndc)::value;
        k_pressure_fix<ND><<<grid_for(bx.count), kThreads, 0, s>>>(g, bx, dt, eps, rho, rhou, E, rho_rec, rhou_rec,
                                                                   E_rec, rho_new, rhou_new, E_new);
    });
    ++g_launches;
}

void internal_mass_gravity(const GridDev& g, const double* rho, int pitch, double central_mass, double* shell,
                           double* g_r, cudaStream_t s)
{
    k_shell_means<<<(g.nx[0] + g.ng + 31) / 32, 32 * kShellWarps, 0, s>>>(g, rho, pitch, shell);
    k_internal_mass_gravity<<<1, kMassThreads, 0, s>>>(g, central_mass, shell, g_r);
    g_launches += 2;
}

void boundaries(const GridDev& g, double* rho, double* rhou, double* E, double* fx, cudaStream_t s)
{
    dispatch_nd(g.ndim, [&](auto ndc) {
        constexpr int ND = decltype(ndc)::value;
        k_fill_ghosts<ND><<<grid_for(g.N), kThreads, 0, s>>>(g, rho, rhou, E, fx);
    });
    ++g_launches;
}

void time_step_inv(const GridDev& g, int ng_eff, const double* rho, const double* u, const double* P,
                   unsigned long long* inv_bits, cudaStream_t s)
{
    const Box bx = make_box(g, ng_eff);
    dispatch_nd(g.ndim, [&](auto ndc) {
        constexpr int ND = decltype(ndc)::value;
        k_time_step<ND><<<grid_for(bx.count), kThreads, 0, s>>>(g, bx, rho, u, P, inv_bits);
    });
    ++g_launches;
}

void min_internal_energy(const GridDev& g, const double* rho, const double* rhou, const double* E,
                         unsigned long long* key, int* nan_flag, cudaStream_t s)
{
    const Box bx = make_box(g, 0);
    dispatch_nd(g.ndim, [&](auto ndc) {
        constexpr int ND = decltype(ndc)::value;
        k_min_evol<ND><<<grid_for(bx.count), kThreads, 0, s>>>(g, bx, rho, rhou, E, key, nan_flag);
    });
    ++g_launches;
}

double decode_min_key(unsigned long long key)
{
    const unsigned long long b = (key >> 63) ? (key & 0x7fffffffffffffffull) : ~key;
    double v;
    static_assert(sizeof(v) == sizeof(b));
    __builtin_memcpy(&v, &b, sizeof(v));
    return v;
}

int integrate_blocks()
{
    return kRedBlocks;
}

void integrate(const GridDev& g, const double* var, double* partials, double* out, cudaStream_t s)
{
    const Box bx = make_box(g, 0);
    k_integrate_partial<<<kRedBlocks, kThreads, 0, s>>>(g, bx, var, partials);
    k_integrate_final<<<1, 32, 0, s>>>(partials, kRedBlocks, out);
    g_launches += 2;
}

} // namespace stage
} // namespace hcl
