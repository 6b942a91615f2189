// march64_fast.cu -- the FP64 march kernels in the fast FP64 forms (compiled
// with FMA contraction; see march1d64.cuh, march2d64.cuh and
// march3d64.cuh).
#include "march1d64.cuh"
#include "march2d64.cuh"
#include "march3d64.cuh"
#include "stages.hpp"

namespace hcl::fused {

bool march1d_fast_valid(const GridDev& g)
{
    return march1d64_valid_t<EOS_PERFECT_GAS_FAST>(g);
}

void configure_march_fast(const GridDev& g)
{
    if (g.ndim == 1) {
        march1d64_configure_t<EOS_PERFECT_GAS_FAST>();
    } else if (march2d64_valid(g)) {
        march64_pick(g, [](auto lim, auto rs) { march2d64_configure_t<decltype(lim)::value, decltype(rs)::value, EOS_PERFECT_GAS_FAST>(); });
    } else if (march3d64_valid(g)) {
        march64_pick(g, [](auto lim, auto rs) {
            march3d64_configure_t<decltype(lim)::value, decltype(rs)::value, EOS_PERFECT_GAS_FAST>();
        });
    }
}

void march1d_fast(const GridDev& g, const StateDev& st0, const StateDev& st1, StepCtl* ctl, const RunParamsDev& rp,
                 int slot0, int steps, cudaStream_t s)
{
    march1d64_launch_t<EOS_PERFECT_GAS_FAST>(g, st0, st1, ctl, rp, slot0, steps, s);
}

void march2d_fast(const GridDev& g, const StateDev& in, const StateDev& out, StepCtl* ctl, const RunParamsDev& rp,
                 int slot, int out_buf, cudaStream_t s)
{
    march64_pick(g, [&](auto lim, auto rs) {
        march2d64_launch_t<decltype(lim)::value, decltype(rs)::value, EOS_PERFECT_GAS_FAST>(g, in, out, ctl, rp, slot, out_buf, s);
    });
}

void march3d_fast(const GridDev& g, const StateDev& in, const StateDev& out, StepCtl* ctl, const RunParamsDev& rp,
                 int slot, int out_buf, cudaStream_t s)
{
    march64_pick(g, [&](auto lim, auto rs) {
        march3d64_launch_t<decltype(lim)::value, decltype(rs)::value, EOS_PERFECT_GAS_FAST>(g, in, out, ctl, rp, slot, out_buf, s);
    });
}

} // namespace hcl::fused
