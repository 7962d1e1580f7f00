// The synthesis passes for the lengths of SL_GROUP_1.
#include "pb_synth_lines.cuh"

namespace pb {
SL_DEFINE_GROUP(1)
}  // namespace pb
