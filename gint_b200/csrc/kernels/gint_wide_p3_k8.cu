// Streaming interpreter kernel (gint_wide.cuh): 3 pool slots of 8 tiles.
#define GINT_WIDE 1
#include "../gint_wide.cuh"
GINT_DEFINE_WIDE_KERNEL(3, 8, 4)
