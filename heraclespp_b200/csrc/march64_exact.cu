// march64_exact.cu -- the FP64 march kernels in the reference's arithmetic
// (compiled with --fmad=false; see march2d64.cuh and march3d64.cuh).
#include "march2d64.cuh"
#include "march3d64.cuh"
#include "stages.hpp"

namespace hcl::fused {

// Cartesian 2-D grids of the perfect gas without scalars or pressure fix
bool march2d64_valid(const GridDev& g)
{
    return g.ndim == 2 && g.geom == GEOM_CARTESIAN && g.eos == EOS_PERFECT_GAS && g.nfx == 0 && !g.pressure_fix;
}

// Cartesian 3-D grids, the same
bool march3d64_valid(const GridDev& g)
{
    return g.ndim == 3 && g.geom == GEOM_CARTESIAN && g.eos == EOS_PERFECT_GAS && g.nfx == 0 && !g.pressure_fix;
}

void configure_march_exact(const GridDev& g)
{
    if (march2d64_valid(g)) {
        march64_pick(g, [](auto lim, auto rs) { march2d64_configure_t<decltype(lim)::value, decltype(rs)::value, EOS_PERFECT_GAS>(); });
    } else if (march3d64_valid(g)) {
        march64_pick(g, [](auto lim, auto rs) {
            march3d64_configure_t<decltype(lim)::value, decltype(rs)::value, EOS_PERFECT_GAS>();
        });
    }
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
