// Row programs of 32-bit floats (gint_rows.cuh): a team of four warps per logical program, one per width value.
#include "../gint_rows.cuh"

extern "C" __global__ void __launch_bounds__(1024) gint_form_rows4_f32(const __grid_constant__ gint::RowsArgs a) { gint::rows_body<4>(a); }
