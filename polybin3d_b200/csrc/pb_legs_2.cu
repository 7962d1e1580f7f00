// The leg passes for the lengths of SL_GROUP_2.
#include "pb_legs.cuh"

namespace pb {
FL_DEFINE_GROUP(2)
}  // namespace pb
