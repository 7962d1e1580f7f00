// The leg passes for the lengths of SL_GROUP_1.
#include "pb_legs.cuh"

namespace pb {
FL_DEFINE_GROUP(1)
}  // namespace pb
