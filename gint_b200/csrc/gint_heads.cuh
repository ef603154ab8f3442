/*
 * gint_heads.cuh -- normalisation of short bfloat16 rows (heads of a projection), four rows per logical program.
 *
 * In 2DT tiles dimension 1 lies along the lanes and the four width values are four rows. A logical program of such a normalisation is
 * a kilobyte; interpreted, its descriptor decode, its 2-byte accesses and its dispatches were 662 warp instructions (heads of 128: 145 us,
 * where the bytes take 41). Here a warp keeps its rows in registers: element 32 c + lane of row w is value [c][w], as in the interpreter,
 * and the sum over the lanes has the interpreter's order, so results are the same bits.
 *
 *   - The next logical program's elements are loaded before the current one is computed.
 *   - A launch of the whole grid takes the logical programs in the order in which they lie in memory (sort_digits in
 *     gint_forms_host.h): neighbouring heads of a token are 256 bytes apart, neighbouring tokens 4 KB.
 *   - The sums of the four rows are reduced together: at the first two steps a lane hands on the half of the values that it does not
 *     go on with (10 shuffles instead of 20, one square root instead of four). The terms of every sum meet in the same order.
 *   - Rows of 128 at 8-byte boundaries have a kernel of their own, four elements per access (heads_body_fours).
 *
 * Measured (one B200, us, cold buffers, interpreter -> here): heads (8, 4096, 16, 128) 145 -> 48.7 (5.5 TB/s; 63 by the kernel of single
 * elements), (8, 8192, 12, 64) 164 -> 55, (2, 4096, 24, 96) 63 -> 25, (3, 777, 12, 80) 19 -> 10. Now 249 warp instructions per logical
 * program, issue slots 0.72 busy. Two logical programs on their way: 51 with four elements per access; no gain for single
 * elements (55 and 57).
 */
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "gint_form_types.h"

namespace gint {

__device__ __forceinline__ float head_value(unsigned short x) { return __uint_as_float((uint32_t)x << 16); }
__device__ __forceinline__ unsigned short head_element(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }

/* offsets (elements) of logical program r in x and y, and its first row: form_offsets (gint_form_types.h) with every digit's numbers at a
 * fixed place in the launch parameters */
struct HeadPlace { uint32_t x, y; int row; };
__device__ __forceinline__ HeadPlace head_place(const HeadsArgs &a, uint32_t r)
{
    HeadPlace p = {0u, 0u, 0};
#pragma unroll
    for (int j = 0; j < kFormDims; j++)
        if (j < (int)a.grid.n_dims) {
            const uint32_t q = form_quotient(a.grid, r, j), b = r - q * a.grid.size[j];
            p.x += b * a.slot[HEADS_X].stride[j];
            p.y += b * a.slot[HEADS_Y].stride[j];
            p.row += (int)(b * a.slot[HEADS_ROW].stride[j]);
            r = q;
        }
    return p;
}

template <int T, bool MASKED> __device__ __forceinline__ void head_load(const unsigned short *p, uint32_t row_stride, int rows, bool last, unsigned short (&x)[T][4])
{
#pragma unroll
    for (int w = 0; w < 4; w++) {
#pragma unroll
        for (int c = 0; c < T; c++) x[c][w] = !MASKED || (w < rows && (c < T - 1 || last)) ? p[32 * c] : (unsigned short)0;
        p += row_stride;
    }
}
template <int T, bool MASKED>
__device__ __forceinline__ void head_store(unsigned short *p, uint32_t row_stride, int rows, bool last, const float (&v)[T][4], const float (&weight)[T], float t)
{
#pragma unroll
    for (int w = 0; w < 4; w++) {
        const float f = __shfl_sync(0xffffffffu, t, 8 * w);
#pragma unroll
        for (int c = 0; c < T; c++) {
            const unsigned short o = head_element(__fmul_rn(weight[c], __fmul_rn(f, v[c][w])));
            if (!MASKED || (w < rows && (c < T - 1 || last))) p[32 * c] = o;
        }
        p += row_stride;
    }
}

/* from the lanes' sums of the four rows: the factor of row w in lanes 8 w .. 8 w + 7 */
__device__ __forceinline__ float head_factor(const HeadsArgs &a, const float (&s)[4], int lane)
{
    /* lanes 16 .. 31 go on with rows 2 and 3, of each half the upper eight lanes with the second of their rows */
    const bool upper = (lane & 16) != 0, second = (lane & 8) != 0;
    const float h0 = __fadd_rn(upper ? s[2] : s[0], __shfl_xor_sync(0xffffffffu, upper ? s[0] : s[2], 16));
    const float h1 = __fadd_rn(upper ? s[3] : s[1], __shfl_xor_sync(0xffffffffu, upper ? s[1] : s[3], 16));
    float t = __fadd_rn(second ? h1 : h0, __shfl_xor_sync(0xffffffffu, second ? h0 : h1, 8));
#pragma unroll
    for (int m = 4; m >= 1; m >>= 1) t = __fadd_rn(t, __shfl_xor_sync(0xffffffffu, t, m));
    return rsqrtf(a.fused ? __fmaf_rn(t, a.factor, a.addend) : __fadd_rn(__fmul_rn(t, a.factor), a.addend));
}

/* T tiles of 32 elements per row */
template <int T> __device__ __forceinline__ void heads_body(const HeadsArgs &a)
{
    const int lane = threadIdx.x & 31;
    const uint32_t warps = blockDim.x >> 5, step = gridDim.x * warps;
    const bool last = 32 * (T - 1) + lane < a.slot[HEADS_X].n, whole = a.slot[HEADS_X].n >= 32 * T;   // (n > 32 (T - 1): only the last tile may lack elements)
    const unsigned short *const x0 = reinterpret_cast<const unsigned short *>(a.slot[HEADS_X].base) + lane;
    unsigned short *const y0 = reinterpret_cast<unsigned short *>(a.slot[HEADS_Y].base) + lane;
    float weight[T];
#pragma unroll
    for (int c = 0; c < T; c++) weight[c] = c < T - 1 || last ? head_value(reinterpret_cast<const unsigned short *>(a.slot[HEADS_W].base)[32 * c + lane]) : 0.0f;
    unsigned short x[T][4];
    HeadPlace next;
    auto load = [&](uint32_t r) {
        next = head_place(a, r);
        if (whole && a.rows - next.row >= 4) head_load<T, false>(x0 + next.x, a.row_stride[HEADS_X], 0, true, x);
        else head_load<T, true>(x0 + next.x, a.row_stride[HEADS_X], a.rows - next.row, last, x);
    };
    uint32_t r = blockIdx.x * warps + (threadIdx.x >> 5);
    if (r < a.count) load(a.first + r);
    for (; r < a.count; r += step) {
        float v[T][4], s[4];
#pragma unroll
        for (int w = 0; w < 4; w++) s[w] = a.init;
#pragma unroll
        for (int c = 0; c < T; c++)
#pragma unroll
            for (int w = 0; w < 4; w++) {
                v[c][w] = head_value(x[c][w]);
                s[w] = __fmaf_rn(v[c][w], v[c][w], s[w]);
            }
        const HeadPlace now = next;
        if (r + step < a.count) load(a.first + r + step);
        const float t = head_factor(a, s, lane);
        if (whole && a.rows - now.row >= 4) head_store<T, false>(y0 + now.y, a.row_stride[HEADS_Y], 0, true, v, weight, t);
        else head_store<T, true>(y0 + now.y, a.row_stride[HEADS_Y], a.rows - now.row, last, v, weight, t);
    }
}

/*
 * Rows of 128 elements at 8-byte boundaries: a lane takes elements 4 l .. 4 l + 3 of every row in one access and keeps the elements of
 * two logical programs on their way. The squares are added in the order of the streaming kernels' vector layout (gint_wide.cuh):
 * per lane elements 4 l .. 4 l + 3, then over the lanes.
 */
__device__ __forceinline__ void head_load_fours(const unsigned short *p, uint32_t row_stride, int rows, uint2 (&x)[4])
{
#pragma unroll
    for (int w = 0; w < 4; w++) {
        x[w] = w < rows ? *reinterpret_cast<const uint2 *>(p) : make_uint2(0u, 0u);
        p += row_stride;
    }
}
__device__ __forceinline__ uint32_t head_pair(float lo, float hi)
{
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %2, %1;" : "=r"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void heads_body_fours(const HeadsArgs &a)
{
    const int lane = threadIdx.x & 31;
    const uint32_t warps = blockDim.x >> 5, step = gridDim.x * warps;
    const unsigned short *const x0 = reinterpret_cast<const unsigned short *>(a.slot[HEADS_X].base) + 4 * lane;
    unsigned short *const y0 = reinterpret_cast<unsigned short *>(a.slot[HEADS_Y].base) + 4 * lane;
    float weight[4];
    {
        const uint2 u = *reinterpret_cast<const uint2 *>(reinterpret_cast<const unsigned short *>(a.slot[HEADS_W].base) + 4 * lane);
        weight[0] = __uint_as_float(u.x << 16); weight[1] = __uint_as_float(u.x & 0xFFFF0000u);
        weight[2] = __uint_as_float(u.y << 16); weight[3] = __uint_as_float(u.y & 0xFFFF0000u);
    }
    uint2 x1[4], x2[4];
    HeadPlace p1, p2;
    uint32_t r = blockIdx.x * warps + (threadIdx.x >> 5);
    auto load = [&](uint32_t at, uint2 (&x)[4], HeadPlace &p) {
        if (at >= a.count) return;
        p = head_place(a, a.first + at);
        head_load_fours(x0 + p.x, a.row_stride[HEADS_X], a.rows - p.row, x);
    };
    load(r, x1, p1);
    load(r + step, x2, p2);
    for (; r < a.count; r += step) {
        float v[4][4], s[4];
#pragma unroll
        for (int w = 0; w < 4; w++) {
            v[0][w] = __uint_as_float(x1[w].x << 16); v[1][w] = __uint_as_float(x1[w].x & 0xFFFF0000u);
            v[2][w] = __uint_as_float(x1[w].y << 16); v[3][w] = __uint_as_float(x1[w].y & 0xFFFF0000u);
            s[w] = a.init;
#pragma unroll
            for (int c = 0; c < 4; c++) s[w] = __fmaf_rn(v[c][w], v[c][w], s[w]);
            x1[w] = x2[w];
        }
        const HeadPlace now = p1;
        p1 = p2;
        load(r + 2u * step, x2, p2);
        const float t = head_factor(a, s, lane);
        unsigned short *y = y0 + now.y;
#pragma unroll
        for (int w = 0; w < 4; w++) {
            const float f = __shfl_sync(0xffffffffu, t, 8 * w);
            float o[4];
#pragma unroll
            for (int c = 0; c < 4; c++) o[c] = __fmul_rn(weight[c], __fmul_rn(f, v[c][w]));
            if (w < a.rows - now.row) *reinterpret_cast<uint2 *>(y) = make_uint2(head_pair(o[0], o[1]), head_pair(o[2], o[3]));
            y += a.row_stride[HEADS_Y];
        }
    }
}

}  // namespace gint

#define GINT_DEFINE_HEADS_KERNEL(T) \
    extern "C" __global__ void __launch_bounds__(256, 4) gint_form_heads_bf16_##T(const __grid_constant__ gint::HeadsArgs a) { gint::heads_body<T>(a); }
#define GINT_DEFINE_HEADS_FOURS_KERNEL \
    extern "C" __global__ void __launch_bounds__(256, 4) gint_form_heads_bf16_fours(const __grid_constant__ gint::HeadsArgs a) { gint::heads_body_fours(a); }
