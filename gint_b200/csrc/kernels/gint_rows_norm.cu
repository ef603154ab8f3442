// Row programs of 32-bit floats (gint_rows.cuh): rows normalised and scaled.
#include "../gint_rows.cuh"
GINT_DEFINE_ROWS_KERNELS(norm)
