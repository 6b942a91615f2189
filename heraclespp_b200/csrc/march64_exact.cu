// march64_exact.cu -- the FP64 march kernels in the reference's arithmetic
// (compiled with --fmad=false; see march1d64.cuh, march2d64.cuh and
// march3d64.cuh).
#include "march1d64.cuh"
#include "march2d64.cuh"
#include "march3d64.cuh"
#include "stages.hpp"

namespace hcl::fused {

bool march1d_exact_valid(const GridDev& g)
{
    return march1d64_valid_t<EOS_PERFECT_GAS>(g);
}

static int sm_count()
{
    static PerDevice cache;
    int dev = 0;
    cudaGetDevice(&dev);
    return cache.get(dev, [dev] {
        int v = 0;
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        return v;
    });
}

// Cartesian 2-D grids of the perfect gas without scalars or pressure fix, from
// more 16 x 16 tiles than one wave of the tile kernel holds (two per SM): a
// strip is at least four row iterations deep, a single tile is quicker (us per
// step, tile and march: 256^2 18.3 and 23.5, 400 x 300 32.4 and 29.3, 512^2
// 59.7 and 45.6)
bool march2d64_valid(const GridDev& g)
{
    const int sms = sm_count();
    return g.ndim == 2 && g.geom == GEOM_CARTESIAN && g.eos == EOS_PERFECT_GAS && g.nfx == 0 && !g.pressure_fix &&
           (int64_t)((g.nx[0] + 15) / 16) * ((g.nx[1] + 15) / 16) > 2 * sms;
}

// Cartesian 3-D grids, the same, where the march's plane steps take less than the
// waves of 8 x 8 x 4 tiles (one per SM): 10.3 us each less 4 against 17.2 us each
// and 6 (in the fast forms 8.0 and 13.2).  A CTA marches at least three planes of
// 30 x 10 columns, so small grids are quicker as tiles (us per step, tile and
// march: 32^3 24 and 50, 48^3 60 and 70, 64^3 126 and 142, 56^3 92 and 80, 80^3 240
// and 183, 128^3 932 and 776, 200 x 100 x 4 61 and 47).
bool march3d64_valid(const GridDev& g)
{
    if (g.ndim != 3 || g.geom != GEOM_CARTESIAN || g.eos != EOS_PERFECT_GAS || g.nfx != 0 || g.pressure_fix) {
        return false;
    }
    const int sms = sm_count();
    const int64_t tiles = (int64_t)((g.nx[0] + 7) / 8) * ((g.nx[1] + 7) / 8) * ((g.nx[2] + 3) / 4);
    const int64_t waves = (tiles + sms - 1) / sms;
    return 5 * waves + 3 > 3 * march3d64_plan(g, sms).cost;
}

void configure_march_exact(const GridDev& g)
{
    if (g.ndim == 1) {
        march1d64_configure_t<EOS_PERFECT_GAS>();
    } else if (march2d64_valid(g)) {
        march64_pick(g, [](auto lim, auto rs) { march2d64_configure_t<decltype(lim)::value, decltype(rs)::value, EOS_PERFECT_GAS>(); });
    } else if (march3d64_valid(g)) {
        march64_pick(g, [](auto lim, auto rs) {
            march3d64_configure_t<decltype(lim)::value, decltype(rs)::value, EOS_PERFECT_GAS>();
        });
    }
}

void march1d_exact(const GridDev& g, const StateDev& st0, const StateDev& st1, StepCtl* ctl, const RunParamsDev& rp,
                 int slot0, int steps, cudaStream_t s)
{
    march1d64_launch_t<EOS_PERFECT_GAS>(g, st0, st1, ctl, rp, slot0, steps, s);
}

void march2d_exact(const GridDev& g, const StateDev& in, const StateDev& out, StepCtl* ctl, const RunParamsDev& rp,
                 int slot, int out_buf, cudaStream_t s)
{
    march64_pick(g, [&](auto lim, auto rs) {
        march2d64_launch_t<decltype(lim)::value, decltype(rs)::value, EOS_PERFECT_GAS>(g, in, out, ctl, rp, slot, out_buf, s);
    });
}

void march3d_exact(const GridDev& g, const StateDev& in, const StateDev& out, StepCtl* ctl, const RunParamsDev& rp,
                 int slot, int out_buf, cudaStream_t s)
{
    march64_pick(g, [&](auto lim, auto rs) {
        march3d64_launch_t<decltype(lim)::value, decltype(rs)::value, EOS_PERFECT_GAS>(g, in, out, ctl, rp, slot, out_buf, s);
    });
}

} // namespace hcl::fused
