// The band-limited chains for the lengths of MR_GROUP_2.
#include "pb_masked.cuh"

namespace pb {
MR_DEFINE_GROUP(2)
}  // namespace pb
