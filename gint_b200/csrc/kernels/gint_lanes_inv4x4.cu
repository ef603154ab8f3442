// The batched 4x4 inverse, compiled ahead of time (gint_lanes.cuh).
#include "../gint_lanes.cuh"
GINT_DEFINE_LANE_KERNEL(inv4x4)
