/*
 * gint_variants.h -- the interpreter kernels shipped inside libgint_b200.so.
 *
 * Each (pool size P, tiles per warp K) pair is compiled separately (gint_b200/csrc/kernels/) and the resulting sm_100a cubin
 * is embedded in the library as a byte array. The host loads the arrays with cudaLibraryLoadData and looks the kernels up by name.
 */
#ifndef GINT_VARIANTS_H
#define GINT_VARIANTS_H

#ifdef __cplusplus
extern "C" {
#endif

#define GINT_DIRECT_VARIANTS(X) X(4, 1) X(4, 2) X(4, 4) X(7, 1) X(7, 2) X(12, 1) X(12, 2)
#define GINT_RF_VARIANTS(X) X(7, 2)       /* virtual registers in shared memory (GINT_RF): the pool is the operand stack alone */
#define GINT_VEC_VARIANTS(X) X(4, 1) X(4, 2)   /* 1-D tiles in the vector layout (GINT_VEC): lane l holds elements 4l..4l+3 */
#define GINT_WIDE_VARIANTS(X) X(3, 8) X(4, 4)   /* streaming kernels (gint_wide.cuh): pool slots, tiles at a time */
#define GINT_WIDEV_VARIANTS(X) X(3, 8) X(4, 4)  /* ... in the vector layout */
#define GINT_INDIRECT_VARIANTS(X) X(12)
#define GINT_CHECKED_VARIANTS(X) X(12)
/* kernels of program forms (gint_forms_host.h), and the files that they are in: X(file, kernel name, index) */
#define GINT_FORM_KERNELS(X)                                                                                                    \
    X(rows_norm, rows1_norm, 0) X(rows_norm, rows4_norm, 1) X(rows_norm_silu_add, rows1_norm_silu_add, 2)                        \
    X(rows_norm_silu_add, rows4_norm_silu_add, 3) X(rows_sum, rows1_sum, 4) X(rows_sum, rows4_sum, 5) X(rows_any, rows1_any, 6)   \
    X(rows_any, rows4_any, 7) X(lanes_bmm4x4, lanes_bmm4x4, 8) X(lanes_inv4x4, lanes_inv4x4, 9) X(heads_bf16, heads_bf16_2, 10)    \
    X(heads_bf16, heads_bf16_3, 11) X(heads_bf16, heads_bf16_4, 12) X(heads_bf16, heads_bf16_fours, 13) X(flat_f32, flat_f32, 14) \
    X(flat_f16, flat_f16, 15) X(flat_bf16, flat_bf16, 16)
#define GINT_N_FORM_KERNELS 17

#define GINT_X_DECL(P, K)                                        \
    extern const unsigned char gint_cubin_direct_##P##_##K[];     \
    extern const unsigned char gint_cubin_direct_##P##_##K##_end[];
GINT_DIRECT_VARIANTS(GINT_X_DECL)
#undef GINT_X_DECL
#define GINT_X_DECL(P, K)                                    \
    extern const unsigned char gint_cubin_rf_##P##_##K[];     \
    extern const unsigned char gint_cubin_rf_##P##_##K##_end[];
GINT_RF_VARIANTS(GINT_X_DECL)
#undef GINT_X_DECL
#define GINT_X_DECL(P, K)                                     \
    extern const unsigned char gint_cubin_vec_##P##_##K[];     \
    extern const unsigned char gint_cubin_vec_##P##_##K##_end[];
GINT_VEC_VARIANTS(GINT_X_DECL)
#undef GINT_X_DECL
#define GINT_X_DECL(P, K)                                      \
    extern const unsigned char gint_cubin_wide_##P##_##K[];     \
    extern const unsigned char gint_cubin_wide_##P##_##K##_end[];
GINT_WIDE_VARIANTS(GINT_X_DECL)
#undef GINT_X_DECL
#define GINT_X_DECL(P, K)                                       \
    extern const unsigned char gint_cubin_widev_##P##_##K[];     \
    extern const unsigned char gint_cubin_widev_##P##_##K##_end[];
GINT_WIDEV_VARIANTS(GINT_X_DECL)
#undef GINT_X_DECL
#define GINT_X_DECL(P)                                     \
    extern const unsigned char gint_cubin_indirect_##P[];   \
    extern const unsigned char gint_cubin_indirect_##P##_end[];
GINT_INDIRECT_VARIANTS(GINT_X_DECL)
#undef GINT_X_DECL
#define GINT_X_DECL(P)                                    \
    extern const unsigned char gint_cubin_checked_##P[];   \
    extern const unsigned char gint_cubin_checked_##P##_end[];
GINT_CHECKED_VARIANTS(GINT_X_DECL)
#undef GINT_X_DECL

#define GINT_X_DECL(file, name, index)                   \
    extern const unsigned char gint_cubin_##file[];       \
    extern const unsigned char gint_cubin_##file##_end[];
GINT_FORM_KERNELS(GINT_X_DECL)
#undef GINT_X_DECL

#ifdef __cplusplus
}
#endif
#endif
