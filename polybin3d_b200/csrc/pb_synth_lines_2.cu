// The synthesis passes for the lengths of SL_GROUP_2.
#include "pb_synth_lines.cuh"

namespace pb {
SL_DEFINE_GROUP(2)
}  // namespace pb
