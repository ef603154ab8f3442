// Row programs of 32-bit floats (gint_rows.cuh): rows summed.
#include "../gint_rows.cuh"
GINT_DEFINE_ROWS_KERNELS(sum)
