// The leg passes of any length, FP32.
#include "pb_legs.cuh"

namespace pb {
cudaError_t fl_any_f32(FlStage stage, const SlParams &p, const FlShells &sh, const SlArgs &a, cudaStream_t s) {
    return fl_launch<float, 0>(stage, p, sh, a, s);
}
}  // namespace pb
