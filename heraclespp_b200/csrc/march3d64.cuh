// march3d64.cuh -- the FP64 3-D fused step (Cartesian grids) as a march along
// z, in the reference's arithmetic (KIND EOS_PERFECT_GAS, bit for bit the tile
// kernel's results) or the fast FP64 forms (EOS_PERFECT_GAS_FAST).
//
// A CTA of W warps owns 30 x (W - 2) output columns and marches them over L
// planes; lane l of warp w holds the Hancock column (i0 - 1 + l, j0 - 1 + w),
// so every thread builds exactly one cell's face states per plane and the
// one-cell halo costs 384/300 of them (8x8x4 tiles: 2.0).  Per plane z:
//   A. the staged FP64 plane z+1 (a 34 x (W + 2) block, copied by cp.async one
//      plane ahead) becomes primitives in a ring of three shared planes;
//   B. Hancock face states of plane z from the ring; the z-face z-1/2 with the
//      column's top state of plane z-1; plane z-1 is complete and stored; the
//      x-faces and the x part of plane z's update;
//   C. the y-faces with the neighbouring row's states;
//   D. the y part of the update (the reference adds x, y, z in this order,
//      godunov_scheme.hpp:114-260).
// The x- and y-face states and what a column carries from plane to plane
// (partial update, lower z-flux, top state) sit in shared memory: kept in
// registers they spill ~1 KB per thread, which the little L1 left beside the
// shared planes cannot hold (1.75 against 1.42 ms below; 16 warps of 128
// registers).  Three barriers per plane order the planes.
//
// What bounds it: FP64 (48 % of the pipe with 45 % of the issue slots; three
// warps per scheduler wait on dependency chains and at the barriers).  A
// 128^2 x 256 step, HLL and Minmod: 4.2 (8x8x4 tiles, a branch per division) ->
// 2.2 (the same tiles with quot64.cuh) -> 1.30 ms (1.42 while the columns past the
// domain's edge, which repeat its last one, asked for a second look each).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "march2d64.cuh"

namespace hcl::fused {

constexpr int kM3Warps = 12;
constexpr int kM3X = 30; // output columns of a CTA
constexpr int kM3Y = kM3Warps - 2;
constexpr int kM3PX = kM3X + 4; // primitive block
constexpr int kM3PY = kM3Y + 4;
constexpr int kM3P = kM3PX * kM3PY;
constexpr int kM3T = 32 * kM3Warps;

struct M3Shared {
    double prim[3][5][kM3P];  // ring of planes
    double stage[5][kM3P];    // FP64 state of the next plane
    double face[4][5][kM3T];  // Hancock states of the plane's x- and y-faces (minus, plus); the
                              // y-minus state gives way to the flux of that face
    double hzT[5][kM3T];      // z-top face state of the previous plane
    double gz[5][kM3T];       // flux of the z-face below the previous plane
    double part[5][kM3T];     // update in progress
    q64::Den hx[kM3PX];       // distance of columns i0 - 2 + k and the next one
    q64::Den hy[kM3PY];
};

template <int LIM, int RS, int KIND>
__global__ void __launch_bounds__(kM3T, 1)
k_march3d64(GridDev g, StateDev in, StateDev out, StepCtl* ctl, RunParamsDev rp, int slot, int out_buf, int ntx, int nty,
            int L)
{
    constexpr bool FAST = KIND == EOS_PERFECT_GAS_FAST;
    constexpr unsigned FULL = 0xffffffffu;
    extern __shared__ __align__(16) unsigned char s_m3[];
    M3Shared& sh = *reinterpret_cast<M3Shared*>(s_m3);
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int w = tid >> 5;
    const Decision dec = decide(ctl, slot, rp);
    if (blockIdx.x == 0 && tid == 0) {
        publish_decision(ctl, dec, rp, slot, out_buf);
    }
    if (dec.noop || dec.neg_dt) {
        return;
    }
    const double dt = dec.dt;
    const double dth = dt / 2;
    const int ng = g.ng, n0 = g.n[0], n1 = g.n[1], n2 = g.n[2];
    const int bx = blockIdx.x % ntx;
    const int by = (blockIdx.x / ntx) % nty;
    const int bz = blockIdx.x / (ntx * nty);
    const int i0 = ng + kM3X * bx;
    const int j0 = ng + kM3Y * by;
    const int zb = ng + L * bz;
    const int ze = min(zb + L, ng + g.nx[2]);
    const int col = i0 - 1 + lane;
    const int row = j0 - 1 + w;
    const bool row_face = row <= ng + g.nx[1];                       // Hancock states needed
    const bool row_out = w >= 1 && w <= kM3Y && row < ng + g.nx[1];
    const bool is_out = row_out && lane >= 1 && lane <= kM3X && col < ng + g.nx[0];
    const exact::Eos e = exact::make_eos(g.gamma, g.gamma_m1, g.mmw, KIND);
    const bool raw = FAST && g.uniform_cart;
    const int64_t plane2 = (int64_t)in.pitch * n1; // doubles per z plane

    // metrics of the thread's column and row (clamped where unused)
    const int cx = min(max(col, 1), n0 - 2);
    const int cy = min(max(row, 1), n1 - 2);
    const double dlx = g.dx[0][cx];
    const double dly = g.dx[1][cy];
    const double gv[3] = {gravity_at(g, cx, 0), gravity_at(g, cx, 1), gravity_at(g, cx, 2)};
    const bool has_g[3] = {g.gravity != GRAV_UNIFORM || g.g[0] != 0.0, g.gravity == GRAV_UNIFORM && g.g[1] != 0.0,
                           g.gravity == GRAV_UNIFORM && g.g[2] != 0.0};
    for (int k = tid; k < kM3PX + kM3PY; k += kM3T) {
        const bool x = k < kM3PX;
        const int d = x ? 0 : 1;
        const int c = min((x ? i0 - 2 + k : j0 - 2 + k - kM3PX), g.n[d] - 2);
        const q64::Den h = raw ? q64::Den{1.0, 1.0} : q64::den((g.dx[d][c] + g.dx[d][c + 1]) / 2);
        (x ? sh.hx[k] : sh.hy[k - kM3PX]) = h;
    }

    // the cells of the primitive block this thread stages and converts
    auto stage_plane = [&](int z) {
        const int zc = min(max(z, 0), n2 - 1);
        for (int p = tid; p < kM3P; p += kM3T) {
            const int i = min(i0 - 2 + p % kM3PX, n0 - 1);
            const int j = min(j0 - 2 + p / kM3PX, n1 - 1);
            const double* src = in.q + zc * plane2 + (int64_t)j * in.pitch + i;
#pragma unroll
            for (int v = 0; v < 5; ++v) {
                const unsigned dst = (unsigned)__cvta_generic_to_shared(&sh.stage[v][p]);
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(src + v * in.plane) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    auto convert_plane = [&](int z) {
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        double(*pr)[kM3P] = sh.prim[z % 3];
        for (int p = tid; p < kM3P; p += kM3T) {
            double q[5], u[5];
#pragma unroll
            for (int v = 0; v < 5; ++v) {
                q[v] = sh.stage[v][p];
            }
            exact::to_prim<3>(e, q, u);
#pragma unroll
            for (int v = 0; v < 5; ++v) {
                pr[v][p] = u[v];
            }
        }
    };
    stage_plane(zb - 2);
    convert_plane(zb - 2);
    stage_plane(zb - 1);
    convert_plane(zb - 1);
    stage_plane(zb);

    const unsigned xm = is_out ? ghost_mask(col, n0, ng, g.bc[0], g.bc[1]) : 0u;
    const unsigned ym = is_out ? ghost_mask(row, n1, ng, g.bc[2], g.bc[3]) : 0u;
    const int pc = (w + 1) * kM3PX + lane + 1; // the thread's cell in the primitive block
    double inv_max = 0.0;
    int64_t bad_cell = -1;

#pragma unroll 1
    for (int z = zb - 1; z <= ze; ++z) {
        // A
        convert_plane(z + 1);
        stage_plane(z + 2);
        __syncthreads();
        // B
        double Uz[2][5]; // z-faces
        double dv, ds[3], dthv;
        if (row_face) {
            const double dlz = g.dx[2][z];
            dv = dlx * dly * dlz;
            ds[0] = dly * dlz;
            ds[1] = dlx * dlz;
            ds[2] = dlx * dly;
            const q64::Den qv = q64::den(dv);
            dthv = q64::quo(dth, qv);
            if (!(q64::within0(dth) && q64::den_ok(dv))) {
                dthv = dth / dv;
            }
            double inc[3][5];
            const double(*pz)[kM3P] = sh.prim[z % 3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                double lo[5], hi[5], U[2][5], F[2][5];
                const double(*pm)[kM3P] = d == 2 ? sh.prim[(z + 2) % 3] : pz;
                const double(*pp)[kM3P] = d == 2 ? sh.prim[(z + 1) % 3] : pz;
                const int off = d == 0 ? 1 : (d == 1 ? kM3PX : 0);
                const auto ld = [&](int k, int v) {
                    return k == 0 ? pm[v][pc - off] : (k == 1 ? pz[v][pc] : pp[v][pc + off]);
                };
                const auto ld_again = [&](int k, int v) {
                    return *(const volatile double*)(k == 0 ? &pm[v][pc - off] : (k == 1 ? &pz[v][pc] : &pp[v][pc + off]));
                };
                q64::Den hL, hR;
                if (d == 0) {
                    hL = sh.hx[lane];
                    hR = sh.hx[lane + 1];
                } else if (d == 1) {
                    hL = sh.hy[w];
                    hR = sh.hy[w + 1];
                } else {
                    hL = raw ? q64::Den{1.0, 1.0} : q64::den((g.dx[2][z - 1] + dlz) / 2);
                    hR = raw ? q64::Den{1.0, 1.0} : q64::den((dlz + g.dx[2][z + 1]) / 2);
                }
                if constexpr (LIM == LIM_CONSTANT) {
#pragma unroll
                    for (int v = 0; v < 5; ++v) {
                        lo[v] = hi[v] = ld(1, v);
                    }
                } else {
                    const double half = raw ? 0.5 : (d == 0 ? dlx : (d == 1 ? dly : dlz)) / 2;
                    exact::faces_ld<5, LIM>(KIND, ld, ld_again, hL, hR, half, lo, hi);
                }
                q64::Range S(e.consts_ok);
                exact::cons_flux_core<3>(e, lo, d, U[0], F[0], S);
                exact::cons_flux_core<3>(e, hi, d, U[1], F[1], S);
                if (!S.ok()) {
#pragma unroll
                    for (int f = 0; f < 2; ++f) {
                        double pt[5], ut[5], ft[5];
#pragma unroll
                        for (int v = 0; v < 5; ++v) {
                            pt[v] = f ? hi[v] : lo[v];
                        }
                        exact::to_cons_flux_slow<3>(e, pt, d, ut, ft);
#pragma unroll
                        for (int v = 0; v < 5; ++v) {
                            U[f][v] = ut[v];
                            F[f][v] = ft[v];
                        }
                    }
                }
#pragma unroll
                for (int v = 0; v < 5; ++v) {
                    inc[d][v] = dthv * ((F[0][v] * ds[d]) - (F[1][v] * ds[d]));
                    if (d == 2) {
                        Uz[0][v] = U[0][v];
                        Uz[1][v] = U[1][v];
                    } else {
                        sh.face[2 * d][v][tid] = U[0][v];
                        sh.face[2 * d + 1][v][tid] = U[1][v];
                    }
                }
            }
            // the predictor's increments of all three dimensions, in order
            auto predict = [&](double* u) {
                const double old[4] = {u[0], u[1], u[2], u[3]};
#pragma unroll
                for (int d = 0; d < 3; ++d) {
#pragma unroll
                    for (int v = 0; v < 5; ++v) {
                        u[v] += inc[d][v];
                    }
                    if (has_g[d]) {
                        u[1 + d] += dth * gv[d] * old[0];
                        u[4] += dth * gv[d] * old[1 + d];
                    }
                }
            };
            predict(Uz[0]);
            predict(Uz[1]);
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                double u[5];
#pragma unroll
                for (int v = 0; v < 5; ++v) {
                    u[v] = sh.face[f][v][tid];
                }
                predict(u);
#pragma unroll
                for (int v = 0; v < 5; ++v) {
                    sh.face[f][v][tid] = u[v];
                }
            }
            __syncwarp();
        }
        if (row_out) {
            if (z >= zb) {
                // z-face z-1/2; plane z-1 is complete
                double top[5], G[5];
#pragma unroll
                for (int v = 0; v < 5; ++v) {
                    top[v] = sh.hzT[v][tid];
                    sh.hzT[v][tid] = Uz[1][v];
                }
                march_riemann<3, RS>(e, top, Uz[0], 2, G);
                if (z > zb && is_out) {
                    const int r = z - 1;
                    const int64_t o = r * plane2 + (int64_t)row * in.pitch + col;
                    const double dlr = g.dx[2][r];
                    const double dvr = dlx * dly * dlr;
                    const q64::Den qv = q64::den(dvr);
                    double dtv = q64::quo(dt, qv);
                    if (!(q64::within0(dt) && q64::den_ok(dvr))) {
                        dtv = dt / dvr;
                    }
                    double qn[5];
#pragma unroll
                    for (int v = 0; v < 5; ++v) {
                        qn[v] = sh.part[v][tid] + dtv * ((sh.gz[v][tid] * ds[2]) - (G[v] * ds[2]));
                    }
                    if (has_g[2]) {
                        qn[3] += dt * gv[2] * in.q[o];
                        qn[4] += dt * gv[2] * in.q[o + 3 * in.plane];
                    }
                    double evol, snd, pn[5];
                    exact::state_prims<3>(e, qn, evol, snd, pn);
                    const double au[3] = {fabs(pn[1]), fabs(pn[2]), fabs(pn[3])};
                    if (!(evol >= 0.0) && bad_cell < 0) {
                        bad_cell = lidx(g, col, row, r);
                    }
#pragma unroll
                    for (int v = 0; v < 5; ++v) {
                        out.q[o + v * out.plane] = qn[v];
                    }
                    auto cfl_max = [&](double cell) {
                        if (isnan(cell)) {
                            inv_max = __longlong_as_double(0x7ff8000000000000ll);
                        } else if (!isnan(inv_max)) {
                            inv_max = inv_max > cell ? inv_max : cell;
                        }
                    };
                    {
                        const double a0 = au[0] + snd, a1 = au[1] + snd, a2 = au[2] + snd;
                        const q64::Den x = q64::den(dlx), y = q64::den(dly), zz = q64::den(dlr);
                        double cell = q64::quo(a0, x) + q64::quo(a1, y) + q64::quo(a2, zz);
                        if (!(q64::within(a0) && q64::within(a1) && q64::within(a2) && q64::den_ok(dlx) &&
                              q64::den_ok(dly) && q64::den_ok(dlr))) {
                            cell = a0 / dlx + a1 / dly + a2 / dlr;
                        }
                        cfl_max(cell);
                    }
                    const unsigned zm =
                        (r < 2 * ng || r >= n2 - 2 * ng) ? ghost_mask(r, n2, ng, g.bc[4], g.bc[5]) : 0u;
                    if ((xm | ym | zm) != 0u) {
                        store_images_3d(out.q, out.plane, out.pitch, n0, n1, n2, ng, col, row, r, xm, ym, zm, qn);
                        // the images' own widths may round differently
                        for (unsigned zk = (zm & 0xffffu) << 1 | 1u; zk; zk &= zk - 1u) {
                            const int kz = __ffs(zk) - 1;
                            const double wz = (au[2] + snd) / g.dx[2][kz ? ghost_slot(kz - 1, n2, ng) : r];
                            for (unsigned yk = (ym & 0xffffu) << 1 | 1u; yk; yk &= yk - 1u) {
                                const int ky = __ffs(yk) - 1;
                                const double wy = (au[1] + snd) / g.dx[1][ky ? ghost_slot(ky - 1, n1, ng) : row];
                                for (unsigned xk = (xm & 0xffffu) << 1 | 1u; xk; xk &= xk - 1u) {
                                    const int kx = __ffs(xk) - 1;
                                    cfl_max((au[0] + snd) / g.dx[0][kx ? ghost_slot(kx - 1, n0, ng) : col] + wy + wz);
                                }
                            }
                        }
                    }
                }
#pragma unroll
                for (int v = 0; v < 5; ++v) {
                    sh.gz[v][tid] = G[v];
                }
            } else {
#pragma unroll
                for (int v = 0; v < 5; ++v) {
                    sh.hzT[v][tid] = Uz[1][v];
                }
            }
            if (z >= zb && z < ze) {
                // x-faces: left face here, right face from the next lane
                double uL[5], uR[5], F[5];
#pragma unroll
                for (int v = 0; v < 5; ++v) {
                    uL[v] = sh.face[1][v][lane ? tid - 1 : tid]; // lane 0 has no left face
                    uR[v] = sh.face[0][v][tid];
                }
                const int64_t o = z * plane2 + (int64_t)min(row, n1 - 1) * in.pitch + min(col, n0 - 1);
                double q[5], qn[5];
#pragma unroll
                for (int v = 0; v < 5; ++v) {
                    q[v] = in.q[o + v * in.plane]; // ahead of the solve, which hides the load
                }
                march_riemann<3, RS>(e, uL, uR, 0, F);
                const double dtv = 2 * dthv; // dt / dv: dt = 2 dth
#pragma unroll
                for (int v = 0; v < 5; ++v) {
                    const double Fr = __shfl_down_sync(FULL, F[v], 1);
                    qn[v] = q[v] + dtv * ((F[v] * ds[0]) - (Fr * ds[0]));
                }
                if (has_g[0]) {
                    qn[1] += dt * gv[0] * q[0];
                    qn[4] += dt * gv[0] * q[1];
                }
#pragma unroll
                for (int v = 0; v < 5; ++v) {
                    sh.part[v][tid] = qn[v];
                }
            }
        }
        __syncthreads();
        // C: the y-face below row w
        const bool in_planes = z >= zb && z < ze;
        if (in_planes && row_face && w >= 1) {
            double dn[5], up[5], G[5];
#pragma unroll
            for (int v = 0; v < 5; ++v) {
                dn[v] = sh.face[3][v][tid - 32];
                up[v] = sh.face[2][v][tid];
            }
            march_riemann<3, RS>(e, dn, up, 1, G);
#pragma unroll
            for (int v = 0; v < 5; ++v) {
                sh.face[2][v][tid] = G[v];
            }
        }
        __syncthreads();
        // D
        if (in_planes && row_out) {
            const int64_t o = z * plane2 + (int64_t)row * in.pitch + min(col, n0 - 1);
            const double dtv = 2 * dthv;
#pragma unroll
            for (int v = 0; v < 5; ++v) {
                sh.part[v][tid] += dtv * ((sh.face[2][v][tid] * ds[1]) - (sh.face[2][v][tid + 32] * ds[1]));
            }
            if (has_g[1]) {
                sh.part[2][tid] += dt * gv[1] * in.q[o];
                sh.part[4][tid] += dt * gv[1] * in.q[o + 2 * in.plane];
            }
        }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    const bool nan_seen = isnan(inv_max);
    const double mx = warp_max_d(nan_seen ? 0.0 : inv_max);
    const unsigned nanv = __ballot_sync(FULL, nan_seen);
    if (lane == 0) {
        atomicMax(&ctl->inv_dt_bits[(slot + 1) % 3], nanv ? 0x7ff8000000000000ull : dbl_bits(mx));
    }
    if (bad_cell >= 0) {
        atomicMin(&ctl->bad_cell, (unsigned long long)bad_cell);
        ctl->err = 4;
        ctl->errflag[(slot + 1) & 1] = 1;
        ctl->final_buf = out_buf;
    }
}

template <int LIM, int RS, int KIND>
int march3d64_configure_t()
{
    static PerDevice cache;
    int dev = 0;
    cudaGetDevice(&dev);
    return cache.get(dev, [dev] {
        int v = 0;
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        cudaFuncSetAttribute(k_march3d64<LIM, RS, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(M3Shared));
        return v;
    });
}

// How `sms` SMs, one CTA each, cover the grid: the planes per CTA with the fewest
// plane steps over all waves (a CTA repeats two planes of face states and stages
// two more), and that count.
struct M3Plan {
    int ntx, nty, L;
    int64_t cost;
};
inline M3Plan march3d64_plan(const GridDev& g, int sms)
{
    M3Plan p{(g.nx[0] + kM3X - 1) / kM3X, (g.nx[1] + kM3Y - 1) / kM3Y, g.nx[2], INT64_MAX};
    const int64_t nt = (int64_t)p.ntx * p.nty;
    for (int c = 1; c <= g.nx[2]; ++c) {
        const int L = (g.nx[2] + c - 1) / c;
        const int64_t ctas = nt * ((g.nx[2] + L - 1) / L);
        const int64_t cost = ((ctas + sms - 1) / sms) * (L + 3);
        if (cost < p.cost) {
            p.cost = cost;
            p.L = L;
        }
    }
    return p;
}

template <int LIM, int RS, int KIND>
void march3d64_launch_t(const GridDev& g, const StateDev& in, const StateDev& out, StepCtl* ctl, const RunParamsDev& rp,
                        int slot, int out_buf, cudaStream_t s)
{
    const int sms = march3d64_configure_t<LIM, RS, KIND>();
    const M3Plan p = march3d64_plan(g, sms);
    const int blocks = p.ntx * p.nty * ((g.nx[2] + p.L - 1) / p.L);
    k_march3d64<LIM, RS, KIND><<<blocks, kM3T, sizeof(M3Shared), s>>>(g, in, out, ctl, rp, slot, out_buf, p.ntx, p.nty, p.L);
    ++g_launches;
}

} // namespace hcl::fused
