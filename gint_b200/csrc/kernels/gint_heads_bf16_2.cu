// Normalisation of bfloat16 rows of 2 tiles of 32 elements (gint_heads.cuh).
#include "../gint_heads.cuh"
GINT_DEFINE_HEADS_KERNEL(2)
