// march2d64.cuh -- the FP64 2-D fused step (Cartesian grids) as a warp-strip
// march, in the reference's arithmetic (KIND EOS_PERFECT_GAS, bit for bit the
// tile kernel's results) or the fast FP64 forms (EOS_PERFECT_GAS_FAST).
//
// A warp owns 28 output columns x L rows; lane l holds column c0 - 2 + l, so
// x-neighbours come from shuffles and lanes 2..29 write.  At row j the warp
// turns the staged FP64 row j+1 into primitives, builds the Hancock face
// states of row j, solves the y-face j-1/2 and finishes row j-1, solves the
// x-faces of row j and adds their part of the update (the reference adds the
// x part first, godunov_scheme.hpp:114-260).  Every primitive, face state and
// flux is computed once per lane.
//
// What bounds it: FP64 (a warp instruction every two cycles per scheduler; 1140
// operations per cell with the halo lanes in the exact form: 0.26 ms for
// 2048^2 at the full rate).  KH 2048^2: 1.02 (tile kernel, a branch per
// division) -> 0.51 ms per step, FP64 pipe 57 % and issue slots 55 % busy, the
// rest waits on dependency chains; the register window (partial update, lower
// flux, top face, row quotients, primitives: 20 doubles) and the straight-line
// groups leave room for three warps per scheduler (one CTA of 12 warps per SM,
// 168 registers).  8 warps: 5 % slower; 16 (128 registers): as fast in the
// exact form, 11 % slower in the fast one.  Fast FP64, 1333 x 1001, Minmod:
// 0.19 -> 0.12 ms.
//
// Gas at rest: zero differences and momenta stay on the straight-line path
// (512^2 blast, Minmod and HLL, 47 us per step as with noise in every cell; 93 us
// when each zero asked for a second look).  A front's tail, momenta from 2^-800
// down to the smallest numbers, is done again out of line; a strip that it crosses
// in every row takes 2.4 times a plain one, and the step waits for it: Gresho
// 512^2 88 us (141 us with plain divisions one by one, tile kernel 99 us).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "fused_step.cuh"
#include "fused_strip2d.cuh"
#include "physics_exact.cuh"

namespace hcl::fused {

constexpr int kMarchLanesOut = 28;
constexpr int kMarchWarps = 12;
constexpr int kMarchRingDoubles = 8 * 4 * 32; // 8 row slots x 4 variables x 32 lanes per warp

// The slopes of a row with tiny or extreme data, by the whole warp (a lane's
// left quotient is its neighbour's): the differences a (x, then y), their
// widths (h_ok: in range), the lower y quotients low.  Gives the quotients q and
// the products s of the slopes and half the widths.
template <int LIM>
static __device__ __noinline__ void slopes_slow(const double* a, q64::Den hx, q64::Den hy, bool h_ok, const double* low,
                                                double dlx, double dly, double* q, double* s)
{
    double Q[8], S[8];
    bool good = h_ok;
#pragma unroll
    for (int v = 0; v < 8; ++v) {
        Q[v] = q64::quo_tiny(a[v], v < 4 ? hx : hy, good);
    }
#pragma unroll
    for (int v = 0; v < 8; ++v) {
        q[v] = Q[v];
    }
    if (!good) {
        for (int v = 0; v < 8; ++v) {
            q[v] = a[v] / (v < 4 ? hx.b : hy.b);
        }
    }
    unsigned bad = 0u;
#pragma unroll
    for (int v = 0; v < 8; ++v) {
        const double R = q[v];
        const double L = v < 4 ? __shfl_up_sync(0xffffffffu, R, 1) : low[v - 4];
        bool pair;
        S[v] = exact::limited_width<LIM>(v < 4 ? dlx : dly) * exact::limited_tiny<LIM>(R, L, pair);
        bad |= (unsigned)!pair << v;
    }
#pragma unroll
    for (int v = 0; v < 8; ++v) {
        s[v] = S[v];
    }
    if (__any_sync(0xffffffffu, bad != 0u)) {
        for (int v = 0; v < 8; ++v) {
            const double L = v < 4 ? __shfl_up_sync(0xffffffffu, q[v], 1) : low[v & 3];
            if (bad >> v & 1u) {
                s[v] = ((v < 4 ? dlx : dly) / 2) * exact::plain::slope(LIM, q[v], L);
            }
        }
    }
}
// the same products in the fast forms, from the quotients
template <int LIM>
static __device__ __noinline__ void slopes_slow_fast(const double* R, const double* L, double wx, double wy, double* s)
{
    for (int v = 0; v < 8; ++v) {
        if (!exact::limited_fast_ok<LIM>(R[v], L[v])) {
            s[v] = (v < 4 ? wx : wy) * exact::plain::slope(LIM, R[v], L[v], EOS_PERFECT_GAS_FAST);
        }
    }
}

// (dl + dl') / 2 across a face; 1 for the fast kind's raw differences on
// uniform grids.  The fast kind takes the plain reciprocal.
template <bool FAST>
__device__ __forceinline__ q64::Den face_width(bool unif, double dl, double dl_p)
{
    if (unif) {
        return q64::Den{1.0, 1.0};
    }
    const double h = (dl + dl_p) / 2;
    return FAST ? q64::Den{h, 1.0 / h} : q64::den(h);
}

template <int ND, int RS>
__device__ __forceinline__ void march_riemann(const exact::Eos& e, const double* cL, const double* cR, int l, double* f)
{
    if constexpr (RS == RS_SPLITTING) {
        exact::plain::riemann<ND>(e, RS, cL, cR, l, f);
    } else {
        exact::riemann_rs<ND, RS>(e, cL, cR, l, f);
    }
}

template <int LIM, int RS, int KIND>
__device__ __forceinline__ void march2d_strip(const GridDev& g, const double* __restrict__ qin, double* __restrict__ qout,
                                              int64_t plane, int pitch, double dt, int sx, int sy, int L,
                                              double& inv_max, int64_t& bad_cell, double (*ring)[4][32])
{
    constexpr bool FAST = KIND == EOS_PERFECT_GAS_FAST;
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int n0 = g.n[0], n1 = g.n[1], ng = g.ng;
    const int c0 = ng + kMarchLanesOut * sx;
    const int col = c0 - 2 + lane;
    const int colc = min(col, n0 - 1);
    const bool out_lane = lane >= 2 && lane < 2 + kMarchLanesOut && col < ng + g.nx[0];
    const int r0 = ng + L * sy;
    const int r1 = min(r0 + L, ng + g.nx[1]);
    const bool in_use = lane < 31 && col < n0 - 1; // the last lane has no right neighbour to look at
    const unsigned xm = out_lane ? ghost_mask(col, n0, ng, g.bc[0], g.bc[1]) : 0u;
    const exact::Eos e = exact::make_eos(g.gamma, g.gamma_m1, g.mmw, KIND);
    const double dth = dt / 2;

    // x metrics of this column (clamped only where the cell is unused)
    const int gx = min(max(col, 1), n0 - 2);
    const int gq = min(col, n0 - 2);
    const double dlx = g.dx[0][gx];
    const double dx2 = g.dx[2][0];
    const bool unif = FAST && g.uniform_cart;
    const q64::Den hx = face_width<FAST>(unif, g.dx[0][gq], g.dx[0][gq + 1]);
    const double wx = unif ? (LIM == LIM_VANLEER ? 1.0 : 0.5) : exact::limited_width<LIM>(dlx);
    const bool hx_ok = FAST || q64::width_ok(hx.b);
    const q64::Den dcol = q64::den(g.dx[0][colc]);
    const double ds1 = dlx * dx2;
    const double gvx = gravity_at(g, gx, 0);
    const double gvy = gravity_at(g, gx, 1);
    const bool has_gx = g.gravity != GRAV_UNIFORM || g.g[0] != 0.0;
    const bool has_gy = g.gravity == GRAV_UNIFORM && g.g[1] != 0.0;

    auto stage_row = [&](int r) {
        const int rc = min(max(r, 0), n1 - 1);
        const int64_t o = (int64_t)rc * pitch + colc;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const unsigned dst = (unsigned)__cvta_generic_to_shared(&ring[r & 7][v][lane]);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(qin + o + plane * v) : "memory");
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    auto row_prim = [&](int r, double* w) {
        double q[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            q[v] = ring[r & 7][v][lane];
        }
        exact::to_prim<2>(e, q, w);
    };

    for (int r = r0 - 2; r <= r0 + 2; ++r) {
        stage_row(r);
    }
    asm volatile("cp.async.wait_group 2;\n" ::: "memory"); // rows r0-2 .. r0 landed
    double wc[4];    // primitives of row j
    double yq[4];    // quotients across the lower y-face of row j
    double hyT[4];   // top face state of row j-1
    double Glo[4];   // flux of the y-face j-3/2
    double qx[4];    // row j-1 with its x part
    double dtodv1 = 0.0; // dt / dv of row j-1
    {
        double wm[4];
        row_prim(r0 - 2, wm);
        row_prim(r0 - 1, wc);
        const q64::Den h = face_width<FAST>(unif, g.dx[1][r0 - 2], g.dx[1][r0 - 1]);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            yq[v] = FAST ? (wc[v] - wm[v]) * h.y : (wc[v] - wm[v]) / h.b;
            hyT[v] = Glo[v] = qx[v] = 0.0;
        }
    }

#pragma unroll 1
    for (int j = r0 - 1; j <= r1; ++j) {
        stage_row(j + 4);
        asm volatile("cp.async.wait_group 2;\n" ::: "memory"); // rows up to j+2 landed
        double wn[4];
        row_prim(j + 1, wn);
        const int jn = min(j + 1, n1 - 1);
        const double dly = g.dx[1][j];
        // one-sided quotients across the x right face and the y upper face of
        // this cell; the left ones come from the next lane and the last row
        double R[8], Lq[8], s[8];
        const q64::Den hy = face_width<FAST>(unif, dly, g.dx[1][jn]);
        const bool h_ok = hx_ok && (FAST || q64::width_ok(hy.b));
        const double wy = unif ? wx : exact::limited_width<LIM>(dly);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const double ax = __shfl_down_sync(FULL, wc[v], 1) - wc[v];
            const double ay = wn[v] - wc[v];
            R[v] = FAST ? ax * hx.y : q64::quo(ax, hx);
            R[4 + v] = FAST ? ay * hy.y : q64::quo(ay, hy);
        }
        q64::Range S(h_ok);
#pragma unroll
        for (int v = 0; v < 8; ++v) {
            Lq[v] = v < 4 ? __shfl_up_sync(FULL, R[v], 1) : yq[v - 4];
            const double w = v < 4 ? wx : wy;
            if constexpr (LIM == LIM_CONSTANT) {
                s[v] = 0.0;
            } else if constexpr (FAST) {
                s[v] = w * exact::limited_fast<LIM>(R[v], Lq[v], S);
            } else {
                s[v] = w * exact::limited_core<LIM>(R[v], Lq[v], S);
            }
        }
        if constexpr (LIM != LIM_CONSTANT) {
            const bool again = in_use && !S.ok();
            if constexpr (FAST) {
                if (again) {
                    double Rt[8], Lt[8], st[8];
#pragma unroll
                    for (int v = 0; v < 8; ++v) {
                        Rt[v] = R[v];
                        Lt[v] = Lq[v];
                        st[v] = s[v];
                    }
                    slopes_slow_fast<LIM>(Rt, Lt, unif ? 0.5 : dlx / 2, unif ? 0.5 : dly / 2, st);
#pragma unroll
                    for (int v = 0; v < 8; ++v) {
                        s[v] = st[v];
                    }
                }
            } else if (__any_sync(FULL, again)) {
                double at[8], lt[4], qt[8], st[8];
                bool low_ok = true;
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    at[v] = __shfl_down_sync(FULL, wc[v], 1) - wc[v];
                    at[4 + v] = wn[v] - wc[v];
                    lt[v] = yq[v];
                    low_ok = low_ok && q64::num_ok(yq[v]);
                }
                if (!low_ok) {
                    // a tiny lower y quotient may be off: row j-1 is still staged
                    double qm[4], wm[4];
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        qm[v] = ring[(j - 1) & 7][v][lane];
                    }
                    exact::to_prim_slow<2, KIND>(e, qm, wm);
                    const double hm = (g.dx[1][j - 1] + dly) / 2;
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        lt[v] = (wc[v] - wm[v]) / hm;
                    }
                }
                slopes_slow<LIM>(at, hx, hy, h_ok, lt, dlx, dly, qt, st);
#pragma unroll
                for (int v = 0; v < 8; ++v) {
                    R[v] = qt[v];
                    s[v] = st[v];
                }
            }
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            yq[v] = R[4 + v];
        }
        // face states (x-left, x-right, y-bottom, y-top) and their fluxes
        double p[4][4], U[4][4], F[4][4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            p[0][v] = wc[v] - s[v];
            p[1][v] = wc[v] + s[v];
            p[2][v] = wc[v] - s[4 + v];
            p[3][v] = wc[v] + s[4 + v];
        }
        {
            q64::Range S(e.consts_ok);
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                exact::cons_flux_core<2>(e, p[f], f >> 1, U[f], F[f], S);
            }
            if (!S.ok()) {
#pragma unroll
                for (int f = 0; f < 4; ++f) {
                    double pt[4], ut[4], ft[4];
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        pt[v] = p[f][v];
                    }
                    exact::to_cons_flux_slow<2>(e, pt, f >> 1, ut, ft);
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        U[f][v] = ut[v];
                        F[f][v] = ft[v];
                    }
                }
            }
        }
        // Hancock predictor (extrapolation_reconstruction.hpp:90-312)
        const double dv = dlx * dly * dx2;
        const double ds0 = dly * dx2;
        const q64::Den qv = q64::den(dv);
        double dthv = q64::quo(dth, qv);
        if (!(q64::within0(dth) && q64::den_ok(dv))) {
            dthv = dth / dv;
        }
        {
            double ix[4], iy[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                ix[v] = dthv * ((F[0][v] * ds0) - (F[1][v] * ds0));
                iy[v] = dthv * ((F[2][v] * ds1) - (F[3][v] * ds1));
            }
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                const double r_old = U[f][0], m0 = U[f][1], m1 = U[f][2];
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    U[f][v] += ix[v];
                }
                if (has_gx) {
                    U[f][1] += dth * gvx * r_old;
                    U[f][3] += dth * gvx * m0;
                }
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    U[f][v] += iy[v];
                }
                if (has_gy) {
                    U[f][2] += dth * gvy * r_old;
                    U[f][3] += dth * gvy * m1;
                }
            }
        }
        // y-face j-1/2, and row j-1 is complete
        double G[4] = {0.0, 0.0, 0.0, 0.0};
        if (j >= r0) {
            march_riemann<2, RS>(e, hyT, U[2], 1, G);
        }
        if (j > r0) {
            const int r = j - 1;
            double qn[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                qn[v] = qx[v] + dtodv1 * ((Glo[v] * ds1) - (G[v] * ds1));
            }
            if (has_gy) {
                qn[2] += dt * gvy * ring[r & 7][0][lane];
                qn[3] += dt * gvy * ring[r & 7][2][lane];
            }
            if (out_lane) {
                double evol, snd, pn[4];
                exact::state_prims<2>(e, qn, evol, snd, pn);
                const double au[2] = {fabs(pn[1]), fabs(pn[2])};
                if (!(evol >= 0.0) && bad_cell < 0) {
                    bad_cell = lidx(g, col, r, 0);
                }
                const int64_t oo = (int64_t)r * pitch + col;
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    qout[oo + plane * v] = qn[v];
                }
                auto cfl_max = [&](double cell) {
                    if (isnan(cell)) {
                        inv_max = __longlong_as_double(0x7ff8000000000000ll);
                    } else if (!isnan(inv_max)) {
                        inv_max = inv_max > cell ? inv_max : cell;
                    }
                };
                {
                    const double ax = au[0] + snd, ay = au[1] + snd;
                    const q64::Den dy = q64::den(g.dx[1][r]);
                    double cell = q64::quo(ax, dcol) + q64::quo(ay, dy);
                    if (!(q64::within(ax) && q64::within(ay) && q64::den_ok(dcol.b) && q64::den_ok(dy.b))) {
                        cell = ax / dcol.b + ay / dy.b;
                    }
                    cfl_max(cell);
                }
                const unsigned ym = (r < 2 * ng || r >= n1 - 2 * ng) ? ghost_mask(r, n1, ng, g.bc[2], g.bc[3]) : 0u;
                if ((xm | ym) != 0u) {
                    store_images_2d(qout, plane, pitch, n0, n1, ng, col, r, xm, ym, qn);
                    // the images' own widths may round differently
                    for (unsigned yb = (ym & 0xffffu) << 1 | 1u; yb; yb &= yb - 1u) {
                        const int ky = __ffs(yb) - 1;
                        const int pj = ky ? ghost_slot(ky - 1, n1, ng) : r;
                        for (unsigned xb = (xm & 0xffffu) << 1 | 1u; xb; xb &= xb - 1u) {
                            const int kx = __ffs(xb) - 1;
                            const int pi = kx ? ghost_slot(kx - 1, n0, ng) : col;
                            cfl_max((au[0] + snd) / g.dx[0][pi] + (au[1] + snd) / g.dx[1][pj]);
                        }
                    }
                }
            }
        }
        // x-faces of row j: left face here, right face from the next lane
        if (j >= r0 && j < r1) {
            double uL[4], Fl[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                uL[v] = __shfl_up_sync(FULL, U[1][v], 1);
            }
            march_riemann<2, RS>(e, uL, U[0], 0, Fl);
            dtodv1 = 2 * dthv; // dt / dv: dt = 2 dth
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const double Fr = __shfl_down_sync(FULL, Fl[v], 1);
                qx[v] = ring[j & 7][v][lane] + dtodv1 * ((Fl[v] * ds0) - (Fr * ds0));
            }
            if (has_gx) {
                qx[1] += dt * gvx * ring[j & 7][0][lane];
                qx[3] += dt * gvx * ring[j & 7][1][lane];
            }
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            hyT[v] = U[3][v];
            Glo[v] = G[v];
            wc[v] = wn[v];
        }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory"); // the ring is reused by the next strip
}

// one step: strips of L rows, `blockDim.x / 32` warps per CTA
template <int LIM, int RS, int KIND>
__global__ void __launch_bounds__(32 * kMarchWarps, 1)
k_march2d64(GridDev g, StateDev in, StateDev out, StepCtl* ctl, RunParamsDev rp, int slot, int out_buf, int L)
{
    extern __shared__ __align__(16) double s_march[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const Decision dec = decide(ctl, slot, rp);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        publish_decision(ctl, dec, rp, slot, out_buf);
    }
    if (dec.noop || dec.neg_dt) {
        return;
    }
    const int ncolw = (g.nx[0] + kMarchLanesOut - 1) / kMarchLanesOut;
    const int nitems = ncolw * ((g.nx[1] + L - 1) / L);
    double inv_max = 0.0;
    int64_t bad_cell = -1;
    auto ring = reinterpret_cast<double (*)[4][32]>(s_march + warp * kMarchRingDoubles);
    const int nw = gridDim.x * (blockDim.x >> 5);
    for (int w = blockIdx.x * (blockDim.x >> 5) + warp; w < nitems; w += nw) {
        march2d_strip<LIM, RS, KIND>(g, in.q, out.q, in.plane, in.pitch, dec.dt, w % ncolw, w / ncolw, L, inv_max,
                                     bad_cell, ring);
    }
    const bool nan_seen = isnan(inv_max);
    const double m = warp_max_d(nan_seen ? 0.0 : inv_max);
    const unsigned nanv = __ballot_sync(0xffffffffu, nan_seen);
    if (lane == 0) {
        atomicMax(&ctl->inv_dt_bits[(slot + 1) % 3], nanv ? 0x7ff8000000000000ull : dbl_bits(m));
    }
    if (bad_cell >= 0) {
        atomicMin(&ctl->bad_cell, (unsigned long long)bad_cell);
        ctl->err = 4;
        ctl->errflag[(slot + 1) & 1] = 1;
        ctl->final_buf = out_buf;
    }
}

// Opts a kernel into its row rings once per device (before any capture);
// returns the device's SM count.
template <int LIM, int RS, int KIND>
int march2d64_configure_t()
{
    static PerDevice cache;
    int dev = 0;
    cudaGetDevice(&dev);
    return cache.get(dev, [dev] {
        int v = 0;
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        cudaFuncSetAttribute(k_march2d64<LIM, RS, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kMarchWarps * kMarchRingDoubles * (int)sizeof(double));
        return v;
    });
}

template <int LIM, int RS, int KIND>
void march2d64_launch_t(const GridDev& g, const StateDev& in, const StateDev& out, StepCtl* ctl, const RunParamsDev& rp,
                        int slot, int out_buf, cudaStream_t s)
{
    // one wave: as many strips per column as the resident warps hold, of at
    // least kMinRows rows (a strip repeats two rows of face states); the CTAs
    // take only the warps that have a strip, so small grids spread over the SMs
    constexpr int kMinRows = 2;
    const int sms = march2d64_configure_t<LIM, RS, KIND>();
    const int ncolw = (g.nx[0] + kMarchLanesOut - 1) / kMarchLanesOut;
    const int per_col = std::max(1, sms * kMarchWarps / ncolw);
    const int L = std::max(std::min(kMinRows, g.nx[1]), (g.nx[1] + per_col - 1) / per_col);
    const int items = ncolw * ((g.nx[1] + L - 1) / L);
    const int warps = std::max(1, std::min(kMarchWarps, (items + sms - 1) / sms));
    const int blocks = std::min(sms, (items + warps - 1) / warps);
    k_march2d64<LIM, RS, KIND><<<blocks, 32 * warps, warps * kMarchRingDoubles * sizeof(double), s>>>(
        g, in, out, ctl, rp, slot, out_buf, L);
    ++g_launches;
}

// f(limiter, solver) with the handle's choices as compile-time constants
template <class F>
void march64_pick(const GridDev& g, F&& f)
{
    auto with_lim = [&](auto lim) {
        if (g.riemann == RS_HLL) {
            f(lim, std::integral_constant<int, RS_HLL>{});
        } else if (g.riemann == RS_HLLC) {
            f(lim, std::integral_constant<int, RS_HLLC>{});
        } else {
            f(lim, std::integral_constant<int, RS_SPLITTING>{});
        }
    };
    if (g.limiter == LIM_VANLEER) {
        with_lim(std::integral_constant<int, LIM_VANLEER>{});
    } else if (g.limiter == LIM_MINMOD) {
        with_lim(std::integral_constant<int, LIM_MINMOD>{});
    } else if (g.limiter == LIM_VANALBADA) {
        with_lim(std::integral_constant<int, LIM_VANALBADA>{});
    } else {
        with_lim(std::integral_constant<int, LIM_CONSTANT>{});
    }
}

} // namespace hcl::fused
