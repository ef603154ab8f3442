// Element-wise programs over contiguous half precision (gint_flat.cuh).
#include "../gint_flat.cuh"
GINT_DEFINE_FLAT_KERNEL(f16, FLAT_F16)
