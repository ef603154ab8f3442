// Normalisation of bfloat16 rows of 128 elements, four elements per lane (gint_heads.cuh).
#include "../gint_heads.cuh"
GINT_DEFINE_HEADS_FOURS_KERNEL
