// Normalisation of short bfloat16 rows (gint_heads.cuh): rows of two to four tiles of 32 elements, and rows of 128 four elements per lane.
#include "../gint_heads.cuh"
GINT_DEFINE_HEADS_KERNEL(2)
GINT_DEFINE_HEADS_KERNEL(3)
GINT_DEFINE_HEADS_KERNEL(4)
GINT_DEFINE_HEADS_FOURS_KERNEL
