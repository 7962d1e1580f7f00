// The leg passes of any length, FP64.
#include "pb_legs.cuh"

namespace pb {
cudaError_t fl_any_f64(FlStage stage, const SlParams &p, const FlShells &sh, const SlArgs &a, cudaStream_t s) {
    return fl_launch<double, 0>(stage, p, sh, a, s);
}
}  // namespace pb
