// The band-limited chains for the lengths of MR_GROUP_1.
#include "pb_masked.cuh"

namespace pb {
MR_DEFINE_GROUP(1)
}  // namespace pb
