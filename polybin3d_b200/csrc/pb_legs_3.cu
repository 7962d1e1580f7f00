// The leg passes for the lengths of SL_GROUP_3.
#include "pb_legs.cuh"

namespace pb {
FL_DEFINE_GROUP(3)
}  // namespace pb
