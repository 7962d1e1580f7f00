// The first synthesis pass of any length, FP32 maps from an FP64 spectrum.
#include "pb_synth_lines.cuh"

namespace pb {
cudaError_t sl_any_f32_src64(SL_ANY_ARGS) { return sl_launch_x<float, double2, 0>(p, a, s); }
}  // namespace pb
