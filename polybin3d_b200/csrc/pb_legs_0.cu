// The leg passes for the lengths of SL_GROUP_0.
#include "pb_legs.cuh"

namespace pb {
FL_DEFINE_GROUP(0)
}  // namespace pb
