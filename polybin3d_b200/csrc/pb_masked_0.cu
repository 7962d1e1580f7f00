// The band-limited chains for the lengths of MR_GROUP_0.
#include "pb_masked.cuh"

namespace pb {
MR_DEFINE_GROUP(0)
}  // namespace pb
