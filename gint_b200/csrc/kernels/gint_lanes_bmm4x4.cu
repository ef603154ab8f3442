// The batched 4x4 product, compiled ahead of time (gint_lanes.cuh).
#include "../gint_lanes.cuh"
GINT_DEFINE_LANE_KERNEL(bmm4x4)
