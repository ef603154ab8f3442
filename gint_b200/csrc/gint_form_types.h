/*
 * gint_form_types.h -- launch arguments of the form kernels, shared by the kernels (gint_rows.cuh) and the host side
 * (gint_forms_host.h).
 *
 * A form is a shape of programs that has a kernel of its own: the host recognises it in the stream with loops (gint_wide_host.h; lane
 * programs in the program as written, instruction for instruction) and a launch hands the kernel what is particular to the program -- slots, sizes, immediates -- as arguments.
 */
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace gint {

typedef unsigned long long u64;

/* A logical program's place in its tensors: the mixed-radix digits of its number, each with a stride per slot. All slots that
 * move share the digits (slots that do not move have strides 0). Division by multiplication: q = (r * magic) >> (31 + shift). */
constexpr int kFormDims = 5;
struct FormGrid {
    uint32_t n_dims;
    uint32_t simple;                 // one digit, and no logical program of the launch reaches its size
    uint32_t size[kFormDims], magic[kFormDims], shift[kFormDims];
    int gather_dim;                  // digit that goes through the row index for the slots in gather_mask; -1: none
    uint32_t gather_mask;
    uint32_t gather_rows;
    const long long *gather_index;
};
struct FormSlot {
    u64 base;
    uint32_t stride[kFormDims];      // elements
    int n;                           // elements of a row (dimension 1 of the block; of row programs no more than their tiles cover); 0: the form has no such operand
    uint32_t area;                   // shared memory: byte offset in the stage, or in the stationary area
    uint32_t stationary;             // the same row for every logical program: staged once
};

__host__ __device__ inline uint32_t form_quotient(const FormGrid &g, uint32_t r, int j)   // r / size[j], r < 2^31
{
    return (uint32_t)(((u64)(r << 1) * g.magic[j]) >> 32) >> g.shift[j];
}
/* offset (elements, modulo 2^32) of logical program r in each of N slots; the gathered digit's row comes in as an argument */
template <int N> __host__ __device__ inline void form_offsets(const FormGrid &g, const FormSlot (&slot)[N], uint32_t r, long long row, uint32_t (&off)[N])
{
    if (g.simple) {   // one digit, which no logical program of the launch wraps
        const uint32_t b = g.gather_dim < 0 ? r : (uint32_t)row;
#pragma unroll
        for (int t = 0; t < N; t++) off[t] = slot[t].stride[0] * (g.gather_mask >> t & 1u ? b : r);
        return;
    }
#pragma unroll
    for (int t = 0; t < N; t++) off[t] = 0;
    for (uint32_t j = 0; j < g.n_dims; j++) {
        const uint32_t q = form_quotient(g, r, (int)j), b = r - q * g.size[j];
        r = q;
#pragma unroll
        for (int t = 0; t < N; t++) off[t] += slot[t].stride[j] * ((int)j == g.gather_dim && ((g.gather_mask >> t) & 1u) ? (uint32_t)row : b);
    }
}

enum { ROWS_SUM = 0, ROWS_SUM_SQUARES, ROWS_FMA_SQUARES };
enum { ROWS_X = 0, ROWS_W, ROWS_R, ROWS_Z, ROWS_N_SLOTS };
enum { ROWS_MAP = 1, ROWS_MAP_W = 2, ROWS_MAP_SILU = 4, ROWS_MAP_R = 8 };
enum { STEPS_ANY = 0, STEPS_TOTAL, STEPS_TOTAL_THEN, STEPS_MEAN };   // the sum over lanes and width values: alone; and steps on single values; and FMulImm, FAddImm, FRSqrt
/* shapes that have kernels of their own: X(name, reduction, map, steps); the last kernels run any */
#define GINT_ROWS_SHAPES(X)                                                                                        \
    X(norm, ROWS_SUM_SQUARES, ROWS_MAP | ROWS_MAP_W, STEPS_MEAN)                                                   \
    X(norm_silu_add, ROWS_SUM_SQUARES, ROWS_MAP | ROWS_MAP_W | ROWS_MAP_SILU | ROWS_MAP_R, STEPS_MEAN)             \
    X(sum, ROWS_SUM, 0, STEPS_TOTAL)                                                                               \
    X(any, -1, -1, STEPS_ANY)
#define GINT_X_SHAPE(name, r, m, s) struct Rows_##name { static constexpr int reduce = r, map = m, steps = s; };
GINT_ROWS_SHAPES(GINT_X_SHAPE)
#undef GINT_X_SHAPE
struct RowsShape { bool fours; };
constexpr RowsShape kRowsShapes[] = {
#define GINT_X_SHAPE(name, r, m, s) {(m) > 0 && (s) == STEPS_MEAN},   // has a pass of four elements at a time
    GINT_ROWS_SHAPES(GINT_X_SHAPE)
#undef GINT_X_SHAPE
};
constexpr int kRowsSteps = 12;
constexpr uint32_t kRowsFold = 0x80;   // step: Dup, FPermW (operand), FAdd

constexpr u64 kRowsWaitNs = 4000000000ull;   // how long a wait for a copy may take where the caller has not said otherwise

struct RowsArgs {
    FormGrid grid;
    FormSlot slot[ROWS_N_SLOTS];
    uint32_t first, count;
    uint32_t tiles, full_tiles;      // tiles of a row; those that are whole in every operand
    uint32_t reduce, map;            // ROWS_SUM ...; 0 or a set of ROWS_MAP...
    float init, silu;
    int store_at;                    // without a map: the running value is stored as a tile at this element
    uint32_t n_steps;
    uint32_t steps;                  // STEPS_...
    uint32_t step[kRowsSteps], operand[kRowsSteps];
    uint32_t depth, stage_bytes, stationary_bytes;
    u64 wait_ns;                     // a wait for a copy that takes longer gives up; 0: every team gives up before its first row
    volatile uint32_t *gave_up;      // host memory: set by a team that gives up
    uint32_t fours;                  // every row of every operand starts at a 16-byte boundary; one length, a multiple of four
};

/* Head programs (gint_heads.cuh): four short rows of bfloat16 elements per logical program, one per width value. */
enum { HEADS_X = 0, HEADS_W, HEADS_Y, HEADS_ROW, HEADS_N_SLOTS };   // HEADS_ROW: not a tensor; its offset is the first row along dimension 2
struct HeadsArgs {
    FormGrid grid;
    FormSlot slot[HEADS_N_SLOTS];
    uint32_t row_stride[HEADS_Y + 1];   // elements between the four rows (W: 0)
    int rows;                        // along dimension 2, in every slot
    uint32_t first, count;
    float init, factor, addend;
    uint32_t fused;                  // the factor and the addend in one fma
};

/* z = [silu](x) [+ y | * y] (gint_flat.cuh): groups [begin, end) of 16 bytes, then `rest` single elements. */
enum { FLAT_SILU = 1, FLAT_ADD = 2, FLAT_MUL = 4 };
struct FlatArgs {
    const void *x, *y;
    void *z;
    uint32_t begin, end, rest;
    uint32_t map;                    // a set of FLAT_...; at most one of FLAT_ADD and FLAT_MUL
    float silu;
};

/* Lane programs (gint_lanes.cuh): tile t of slot s covers rows 32 t .. 32 t + 31 of rows[s], each `stride` elements apart. */
struct LaneArgs {
    u64 base[8];
    uint32_t stride[8];
    int rows[8];
    uint32_t first, count;           // tiles
    uint32_t depth;
};
constexpr uint32_t kLaneTileBytes = 2048;   // 32 rows of 16 floats

}  // namespace gint
