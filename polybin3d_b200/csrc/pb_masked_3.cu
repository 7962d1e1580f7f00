// The band-limited chains for the lengths of MR_GROUP_3.
#include "pb_masked.cuh"

namespace pb {
MR_DEFINE_GROUP(3)
}  // namespace pb
