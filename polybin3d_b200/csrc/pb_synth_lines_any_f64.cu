// The synthesis passes of any length, FP64.
#include "pb_synth_lines.cuh"

namespace pb {
cudaError_t sl_any_f64(SL_ANY_ARGS) { return sl_launch<double, double2, 0>(stage, p, a, s); }
}  // namespace pb
