// Row programs of 32-bit floats (gint_rows.cuh): rows of any shape.
#include "../gint_rows.cuh"
GINT_DEFINE_ROWS_KERNELS(any)
