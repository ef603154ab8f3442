// Row programs of 32-bit floats (gint_rows.cuh): rows normalised, scaled, through SiLU, plus a residual.
#include "../gint_rows.cuh"
GINT_DEFINE_ROWS_KERNELS(norm_silu_add)
