// march1d64.cuh -- many FP64 1-D steps in one launch: a cluster of up to 16
// CTAs keeps the whole domain in shared memory.
//
// What bounds a 1-D run: latency.  1024 cells are ~5e5 FP64 operations per
// step, under 0.1 us of the card, but a step is a chain of ~200 dependent FP64
// operations (slope, predictor, Riemann problem, update, conversion, CFL) that
// ends in a maximum over the domain, and as one kernel per step it also waits
// for a launch and for global memory.  Here each CTA owns a run of cells, one
// per thread; a step costs three CTA barriers and one cluster barrier, across
// which neighbours pass the primitives of two cells each way and every warp its
// largest 1/dt, all through distributed shared memory.  Cycles of a step: the
// maximum and dt 1000, face states 1650, Riemann problem 1050, update and next
// primitives ~1000, exchange and cluster barrier ~2000.
//
// us per step, FP64 / fast FP64, one kernel per step against this: 1024 cells
// 7.6 / 6.9 -> 3.2 / 3.0, 4096 cells 7.8 / 6.9 -> 4.1 / 3.5, 8192 cells 8.1 /
// 6.9 -> 6.0 / 4.9 (one SM's FP64 pipe takes over: 512 cells per CTA), which is
// why the line lies there.
//
// The arithmetic per cell is the tile kernel's (KIND EOS_PERFECT_GAS: the
// reference's, bit for bit; EOS_PERFECT_GAS_FAST: the fast FP64 forms), the
// time-loop control is decide_values().
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "fused_step.cuh"
#include "physics_exact.cuh"

namespace hcl::fused {

constexpr int kM1MaxCtas = 16;
constexpr int kM1MaxChunk = 512; // cells of a CTA
constexpr int kM1MaxThreads = 288;
constexpr int kM1MaxWarps = kM1MaxThreads / 32;

// Shared memory of one CTA, [k] local cell k - 2 of the run (two cells of
// halo on each side).
struct M1Shared {
    // largest 1/dt (bits) of each warp of the cluster, by step parity; all ones
    // where the warp met an invalid state
    unsigned long long top[2][kM1MaxCtas * (kM1MaxWarps + 1)];
    // What the run sends each step: own cell `from` to cell `to` of run `rank`
    // (halos of the neighbours and, through the boundary conditions, ghost
    // cells), and the ghost cells it fills, for their share of the CFL.
    struct Send {
        int from, rank, to, flip;
    } send[4 * kM1MaxCtas];
    int nsend;
    int ghost_from[8];
    q64::Den ghost_w[8];
    int nghost;
    double a[kM1MaxChunk + 4]; // |u| + c of the new state
    double q[3][kM1MaxChunk + 4];    // conservative state of the run's own cells
    double p[2][3][kM1MaxChunk + 4]; // primitives, by step parity
    double fl[3][kM1MaxChunk + 4];   // predicted left and right face states
    double fr[3][kM1MaxChunk + 4];
    double flux[3][kM1MaxChunk + 4]; // of the left face
    double dl[kM1MaxChunk + 4];
    double ds[kM1MaxChunk + 5]; // left face areas
    q64::Den h[kM1MaxChunk + 4]; // distance to the next cell
    q64::Den dv[kM1MaxChunk + 4];
    q64::Den cw[kM1MaxChunk + 4]; // cell width in the CFL
};

template <int KIND>
__device__ __forceinline__ void m1_faces(int lim, const double* m, const double* c, const double* p, const q64::Den& hL,
                                         const q64::Den& hR, double half, double* lo, double* hi)
{
    if (lim == LIM_VANLEER) {
        exact::faces_den<3, LIM_VANLEER>(KIND, m, c, p, hL, hR, half, lo, hi);
    } else if (lim == LIM_MINMOD) {
        exact::faces_den<3, LIM_MINMOD>(KIND, m, c, p, hL, hR, half, lo, hi);
    } else if (lim == LIM_VANALBADA) {
        exact::faces_den<3, LIM_VANALBADA>(KIND, m, c, p, hL, hR, half, lo, hi);
    } else {
#pragma unroll
        for (int v = 0; v < 3; ++v) {
            lo[v] = hi[v] = c[v];
        }
    }
}

// `steps` steps from buffer `counter & 1` (the state of step `counter`), fewer
// when the run stops.  st0/st1: the two state buffers.
template <int KIND>
__global__ void __launch_bounds__(kM1MaxThreads, 1) k_march1d64(GridDev g, StateDev st0, StateDev st1, StepCtl* ctl, RunParamsDev rp, int slot0, int steps,
                            int chunk)
{
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char s_m1[];
    M1Shared& sh = *reinterpret_cast<M1Shared*>(s_m1);
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    const int nr = (int)cl.num_blocks();
    const int tid = threadIdx.x, nt = blockDim.x;
    const int lane = tid & 31;
    const int ng = g.ng, n = g.n[0], end = ng + g.nx[0];
    const int first = ng + rank * chunk; // global index of the run's first cell
    const int ncell = max(0, min(chunk, end - first));
    const exact::Eos e = exact::make_eos(g.gamma, g.gamma_m1, g.mmw, KIND);
    const bool raw = KIND == EOS_PERFECT_GAS_FAST && g.uniform_cart;
    const bool sph = g.geom == GEOM_SPHERICAL;
    const bool has_g = g.gravity != GRAV_UNIFORM || g.g[0] != 0.0;

    const int p0 = slot0 & 1;
    double t = ctl->t[p0];
    int iter = ctl->iter[p0], toid = ctl->time_output_id[p0], ioid = ctl->iter_output_id[p0];
    bool noop = ctl->stop[p0] || ctl->errflag[p0];
    const bool noop_at_start = noop;
    const int err_at_start = ctl->errflag[p0];
    const unsigned long long inv0 = ctl->inv_dt_bits[slot0 % 3];

    // state and metrics of the run and its halo
    const StateDev in = p0 ? st1 : st0;
    for (int k = tid; k < ncell + 4; k += nt) {
        const int i = first - 2 + k;
        double q[3], p[3];
#pragma unroll
        for (int v = 0; v < 3; ++v) {
            q[v] = in.q[i + in.plane * v];
        }
        exact::to_prim<1>(e, q, p);
#pragma unroll
        for (int v = 0; v < 3; ++v) {
            sh.q[v][k] = q[v];
            sh.p[0][v][k] = p[v];
        }
        const int c = min(max(i, 1), n - 2);
        const double dl = g.dx[0][c];
        sh.dl[k] = dl;
        const double hn = i < n - 1 ? (g.dx[0][i] + g.dx[0][i + 1]) / 2 : dl;
        sh.h[k] = raw ? q64::Den{1.0, 1.0} : q64::Den{hn, 1.0 / hn};
        const double dv = sph ? g.dv[c] : dl * g.dx[1][0] * g.dx[2][0];
        sh.dv[k] = q64::Den{dv, 1.0 / dv};
        sh.ds[k] = sph ? g.ds[min(i, n - 1)] : 1 * g.dx[1][0] * g.dx[2][0];
        const double w = g.dx[0][min(i, n - 1)];
        sh.cw[k] = q64::Den{w, 1.0 / w};
    }
    if (tid == 0) {
        sh.nsend = sh.nghost = 0;
    }
    __syncthreads();
    if (tid < 4 * nr) {
        const int r = tid >> 2, side = tid & 3;
        const int nl = min(chunk, end - (ng + r * chunk));
        const int to = side < 2 ? side : nl + side;
        int flip;
        const int i = bc_source(ng + r * chunk - 2 + to, n, ng, g.bc[0], g.bc[1], &flip);
        if ((i - ng) / chunk == rank) {
            sh.send[atomicAdd(&sh.nsend, 1)] = M1Shared::Send{i - first + 2, r, to, flip};
        }
    }
    if (tid < 2 * ng) {
        const int pos = ghost_slot(tid, n, ng);
        int flip;
        const int i = bc_source(pos, n, ng, g.bc[0], g.bc[1], &flip);
        if ((i - ng) / chunk == rank) {
            const int e2 = atomicAdd(&sh.nghost, 1);
            sh.ghost_from[e2] = i - first + 2;
            sh.ghost_w[e2] = q64::Den{g.dx[0][pos], 1.0 / g.dx[0][pos]};
        }
    }
    if (tid == 0) {
        sh.ds[ncell + 4] = sph ? g.ds[min(first + ncell + 2, n - 1)] : 1 * g.dx[1][0] * g.dx[2][0];
    }
    cl.sync();
    // the cluster's largest value of a parity, the same in every thread
    const int nw = nt >> 5;
    const int nslot = nr * (nw + 1);
    auto cluster_top = [&](int par) {
        unsigned long long m = 0ull;
        for (int k = lane; k < nslot; k += 32) {
            m = max(m, sh.top[par][k]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        }
        return m;
    };
    unsigned long long inv = inv0;

    int done = 0;
    bool stop = false, neg = false, invalid = false;
    double last_dt = 0.0;
    for (int s = 0; s < steps && !noop; ++s) {
        const Decision dec = decide_values(t, iter, toid, ioid, inv, rp);
        toid = dec.toid_next;
        ioid = dec.ioid_next;
        stop = dec.stop != 0;
        last_dt = dec.dt;
        if (dec.neg_dt) {
            neg = true;
            break;
        }
        const double dt = dec.dt;
        const double dth = dt / 2;
        if (rank == 0 && tid == 0 && rp.dt_log && iter < rp.dt_log_cap) {
            rp.dt_log[iter] = dt;
        }
        const int b = s & 1;
        // Hancock face states of the run and one cell on each side
        for (int k = 1 + tid; k < ncell + 3; k += nt) {
            double m[3], c[3], p[3], f[2][3], U[2][3], F[2][3];
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                m[v] = sh.p[b][v][k - 1];
                c[v] = sh.p[b][v][k];
                p[v] = sh.p[b][v][k + 1];
            }
            m1_faces<KIND>(g.limiter, m, c, p, sh.h[k - 1], sh.h[k], raw ? 0.5 : sh.dl[k] / 2, f[0], f[1]);
            exact::to_cons_flux<1>(e, f[0], 0, U[0], F[0]);
            exact::to_cons_flux<1>(e, f[1], 0, U[1], F[1]);
            double dtodv = q64::quo(dth, sh.dv[k]);
            if (!(q64::within0(dth) && q64::den_ok(sh.dv[k].b))) {
                dtodv = dth / sh.dv[k].b;
            }
            const double dsc = sh.ds[k], dsp = sph ? sh.ds[k + 1] : dsc;
            const double gd = gravity_at(g, min(max(first - 2 + k, 1), n - 2), 0);
#pragma unroll
            for (int f2 = 0; f2 < 2; ++f2) {
                const double r_old = U[f2][0], m_old = U[f2][1];
#pragma unroll
                for (int v = 0; v < 3; ++v) {
                    U[f2][v] += dtodv * ((F[0][v] * dsc) - (F[1][v] * dsp));
                }
                if (sph) {
                    U[f2][1] += exact::src_grad_pres(dtodv, f[0][2], f[1][2], dsc, dsp);
                }
                if (has_g) {
                    U[f2][1] += dth * gd * r_old;
                    U[f2][2] += dth * gd * m_old;
                }
            }
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                sh.fl[v][k] = U[0][v];
                sh.fr[v][k] = U[1][v];
            }
        }
        __syncthreads();
        for (int k = 2 + tid; k < ncell + 3; k += nt) {
            double cL[3], cR[3], F[3];
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                cL[v] = sh.fr[v][k - 1];
                cR[v] = sh.fl[v][k];
            }
            exact::riemann<1>(e, g.riemann, cL, cR, 0, F);
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                sh.flux[v][k] = F[v];
            }
        }
        __syncthreads();
        // update, health check, CFL; the new primitives to every run that reads them
        double inv_max = 0.0;
        bool bad = false;
        auto cfl_max = [&](double cell) {
            if (isnan(cell)) {
                inv_max = __longlong_as_double(0x7ff8000000000000ll);
            } else if (!isnan(inv_max)) {
                inv_max = inv_max > cell ? inv_max : cell;
            }
        };
        for (int k = 2 + tid; k < ncell + 2; k += nt) {
            const int i = first - 2 + k;
            double qn[3], q[3];
            double dtodv = q64::quo(dt, sh.dv[k]);
            if (!(q64::within0(dt) && q64::den_ok(sh.dv[k].b))) {
                dtodv = dt / sh.dv[k].b;
            }
            const double dsc = sh.ds[k], dsp = sph ? sh.ds[k + 1] : dsc;
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                q[v] = sh.q[v][k];
                qn[v] = q[v] + dtodv * ((sh.flux[v][k] * dsc) - (sh.flux[v][k + 1] * dsp));
            }
            if (sph) {
                double vL[3], vR[3], pl[3], pr[3];
#pragma unroll
                for (int v = 0; v < 3; ++v) {
                    vL[v] = sh.fl[v][k];
                    vR[v] = sh.fr[v][k];
                }
                exact::to_prim<1>(e, vL, pl);
                exact::to_prim<1>(e, vR, pr);
                qn[1] += exact::src_grad_pres(dtodv, pl[2], pr[2], dsc, dsp);
            }
            if (has_g) {
                const double gd = gravity_at(g, i, 0);
                qn[1] += dt * gd * q[0];
                qn[2] += dt * gd * q[1];
            }
            double evol, snd, pn[3];
            exact::state_prims<1>(e, qn, evol, snd, pn); // the next step's primitives too
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                sh.q[v][k] = qn[v];
            }
            if (!(evol >= 0.0)) {
                bad = true;
                atomicMin(&ctl->bad_cell, (unsigned long long)i);
            }
            const double a = fabs(pn[1]) + snd;
            double cell = q64::quo(a, sh.cw[k]);
            if (!(q64::within(a) && q64::den_ok(sh.cw[k].b))) {
                cell = a / sh.cw[k].b;
            }
            sh.a[k] = a;
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                sh.p[b ^ 1][v][k] = pn[v];
            }
            cfl_max(cell);
        }
        // the warp's largest 1/dt to every CTA, each in its own slot
        auto publish = [&](int slot) {
            const unsigned nanv = __ballot_sync(0xffffffffu, isnan(inv_max));
            const unsigned badv = __ballot_sync(0xffffffffu, bad);
            const double mx = warp_max_d(isnan(inv_max) ? 0.0 : inv_max);
            if (lane < nr) {
                M1Shared* o = lane == rank ? &sh : cl.map_shared_rank(&sh, lane);
                o->top[b][rank * (nw + 1) + slot] = badv ? ~0ull : (nanv ? 0x7ff8000000000000ull : dbl_bits(mx));
            }
        };
        publish(tid >> 5);
        __syncthreads();
        if ((tid >> 5) == nw - 1) {
            // the last warp, which has the fewest cells, sends the run's edges
            for (int x = lane; x < sh.nsend; x += 32) {
                const M1Shared::Send d = sh.send[x];
                M1Shared* o = d.rank == rank ? &sh : cl.map_shared_rank(&sh, d.rank);
                const double ux = sh.p[b ^ 1][1][d.from];
                o->p[b ^ 1][0][d.to] = sh.p[b ^ 1][0][d.from];
                o->p[b ^ 1][1][d.to] = d.flip ? -ux : ux;
                o->p[b ^ 1][2][d.to] = sh.p[b ^ 1][2][d.from];
            }
            inv_max = 0.0;
            bad = false;
            if (lane < sh.nghost) {
                const double a = sh.a[sh.ghost_from[lane]];
                const q64::Den w = sh.ghost_w[lane];
                double cell = q64::quo(a, w);
                if (!(q64::within(a) && q64::den_ok(w.b))) {
                    cell = a / w.b;
                }
                cfl_max(cell);
            }
            publish(nw);
        }
        t = dec.t + dt;
        iter = dec.iter + 1;
        ++done;
        cl.sync();
        inv = cluster_top(b);
        invalid = inv == ~0ull;
        noop = stop || invalid;
    }

    // the final state with its ghost cells, and the control block as `steps`
    // single steps leave it
    if (done > 0) {
        const StateDev out = ((p0 + done) & 1) ? st1 : st0;
        for (int k = 2 + tid; k < ncell + 2; k += nt) {
            const int i = first - 2 + k;
            const double q[3] = {sh.q[0][k], sh.q[1][k], sh.q[2][k]};
            const unsigned xm = ghost_mask(i, n, ng, g.bc[0], g.bc[1]);
            for (unsigned xb = (xm & 0xffffu) << 1 | 1u; xb; xb &= xb - 1u) {
                const int kx = __ffs(xb) - 1;
                const int pos = kx ? ghost_slot(kx - 1, n, ng) : i;
                const bool flip = kx && ((xm >> (15 + kx)) & 1u);
                out.q[pos] = q[0];
                out.q[pos + out.plane] = flip ? -q[1] : q[1];
                out.q[pos + 2 * out.plane] = q[2];
            }
        }
    }
    if (rank == 0 && tid == 0) {
        const int q = (slot0 + steps) & 1;
        if (invalid) {
            ctl->err = 4; // HCL_ERR_INVALID_STATE
        }
        if (neg) {
            ctl->err = 5; // HCL_ERR_NEGATIVE_DT, main.cpp:368-371
        }
        const bool early = noop_at_start || done + (neg ? 1 : 0) < steps; // steps that did nothing followed
        ctl->t[q] = t;
        ctl->iter[q] = iter;
        ctl->time_output_id[q] = toid;
        ctl->iter_output_id[q] = ioid;
        ctl->stop[q] = stop || early;
        ctl->errflag[q] = invalid || neg || err_at_start;
        if (!noop_at_start) {
            ctl->last_dt = last_dt;
            if (stop || invalid || neg) {
                ctl->final_buf = (p0 + done) & 1;
            }
        }
        ctl->inv_dt_bits[(slot0 + steps) % 3] = inv;
        ctl->inv_dt_bits[(slot0 + steps + 1) % 3] = 0ull;
        ctl->inv_dt_bits[(slot0 + steps + 2) % 3] = 0ull;
    }
    cl.sync(); // no CTA leaves while another may still write to its shared memory
}

inline cudaLaunchConfig_t march1d64_config(int ctas, int threads, cudaStream_t s, cudaLaunchAttribute* at)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = sizeof(M1Shared);
    cfg.stream = s;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

template <int KIND>
bool march1d64_configure_t()
{
    static PerDevice cache;
    int dev = 0;
    cudaGetDevice(&dev);
    return cache.get(dev, [] {
        // the largest cluster must fit this device (or the part of it in use)
        cudaLaunchAttribute at[1];
        cudaLaunchConfig_t cfg = march1d64_config(kM1MaxCtas, kM1MaxThreads, nullptr, at);
        int clusters = 0;
        const bool ok = cudaFuncSetAttribute(k_march1d64<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(M1Shared)) == cudaSuccess &&
                        cudaFuncSetAttribute(k_march1d64<KIND>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                            cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&clusters, k_march1d64<KIND>, &cfg) == cudaSuccess && clusters > 0;
        cudaGetLastError();
        return ok ? 1 : 0;
    }) != 0;
}

// Perfect-gas 1-D domains without scalars or pressure fix, with a gravity table
// that does not change from step to step, up to 16 CTAs' cells, where this kind's
// kernel can be launched
template <int KIND>
bool march1d64_valid_t(const GridDev& g)
{
    return g.ndim == 1 && g.eos == EOS_PERFECT_GAS && g.nfx == 0 && !g.pressure_fix &&
           g.gravity != GRAV_INTERNAL_MASS && g.nx[0] <= kM1MaxCtas * kM1MaxChunk && march1d64_configure_t<KIND>();
}

// cells per CTA: the smallest multiple of 32 that 16 CTAs cover the domain with
inline int march1d64_chunk(const GridDev& g)
{
    const int c = (g.nx[0] + kM1MaxCtas - 1) / kM1MaxCtas;
    return std::max(32, (c + 31) / 32 * 32);
}

template <int KIND>
void march1d64_launch_t(const GridDev& g, const StateDev& st0, const StateDev& st1, StepCtl* ctl, const RunParamsDev& rp,
                        int slot0, int steps, cudaStream_t s)
{
    const int chunk = march1d64_chunk(g);
    const int ctas = (g.nx[0] + chunk - 1) / chunk;
    // one thread per cell and the halo's in the same round
    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t cfg = march1d64_config(ctas, std::min(chunk, kM1MaxThreads - 32) + 32, s, at);
    cudaLaunchKernelEx(&cfg, k_march1d64<KIND>, g, st0, st1, ctl, rp, slot0, steps, chunk);
    ++g_launches;
}

} // namespace hcl::fused
