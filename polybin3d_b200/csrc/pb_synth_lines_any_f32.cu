// The synthesis passes of any length, FP32.
#include "pb_synth_lines.cuh"

namespace pb {
cudaError_t sl_any_f32(SL_ANY_ARGS) { return sl_launch<float, float2, 0>(stage, p, a, s); }
}  // namespace pb
