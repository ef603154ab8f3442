// Streaming interpreter kernel (gint_wide.cuh): 4 pool slots of 4 tiles.
#define GINT_WIDE 1
#include "../gint_wide.cuh"
GINT_DEFINE_WIDE_KERNEL(4, 4, 5)
