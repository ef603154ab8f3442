// Element-wise programs over contiguous bfloat16 (gint_flat.cuh).
#include "../gint_flat.cuh"
GINT_DEFINE_FLAT_KERNEL(bf16, FLAT_BF16)
