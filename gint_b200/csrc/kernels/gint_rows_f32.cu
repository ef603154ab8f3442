// Row programs of 32-bit floats (gint_rows.cuh): one warp per logical program, and one warp per width value.
#include "../gint_rows.cuh"

extern "C" __global__ void __launch_bounds__(768) gint_form_rows_f32(const __grid_constant__ gint::RowsArgs a) { gint::rows_body<1>(a); }
