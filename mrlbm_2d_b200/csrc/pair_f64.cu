// pair_f64.cu -- FP64 two-step instantiations.  Built with -fmad=false like step_f64.cu: every
// product and sum rounds separately, so a pair gives the bits of two single steps.
#include "step_fp64.cuh"
#include "step_pair.cuh"

namespace mrlbm {

// Four warps of one strip: two strips per warp halve the warps the ring has room for and were slower
// (4099 x 1023: 72 us per step against 62), six ring rows instead of five as well (64 us).
int launch_pair_f64(const StepParams<double>& p1, const StepParams<double>& p2, const PairPlan& plan, bool flip, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    return (p1.fstat || p1.body) ? launch_pair<fp64::Physics, true, 4, 1, 5, PAIR_MINB>(p1, p2, plan, flip, s)
                                 : launch_pair<fp64::PhysicsLean, false, 4, 1, 5, PAIR_MINB>(p1, p2, plan, flip, s);
}

}  // namespace mrlbm
