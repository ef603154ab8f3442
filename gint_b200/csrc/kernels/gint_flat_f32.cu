// Element-wise programs over contiguous 32-bit floats (gint_flat.cuh).
#include "../gint_flat.cuh"
GINT_DEFINE_FLAT_KERNEL(f32, FLAT_F32)
