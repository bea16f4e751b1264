// pair_f32.cu -- FP32 two-step instantiations (contraction allowed, as in step_f32.cu).
#include "step_fp32.cuh"
#include "step_pair.cuh"

namespace mrlbm {

// Four warps of two strips, whose nodes go through the packed arithmetic two at a time: one strip
// per warp (eight warps) was slower (4099 x 1023: 39 us per step against 36).
int launch_pair_f32(const StepParams<float>& p1, const StepParams<float>& p2, const PairPlan& plan, bool flip, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    return (p1.fstat || p1.body) ? launch_pair<fp32::Physics, true, 4, 2, 6, PAIR_MINB>(p1, p2, plan, flip, s)
                                 : launch_pair<fp32::PhysicsLean, false, 4, 2, 6, PAIR_MINB>(p1, p2, plan, flip, s);
}

}  // namespace mrlbm
