/*
 * gint_flat.cuh -- z = [silu](x) [+ y | * y] over contiguous elements, in groups of 16 bytes.
 *
 * On the streaming kernels a SiLU and a product took 162 warp instructions per 128 values, most of them the exponential and a division
 * with a branch per element; short launches on the tile kernels pay a block's set-up and six dependent dispatches for one tile. Here the
 * quotient is that of gint_silu.cuh and everything else is one loop over 16-byte accesses; a warp's groups of one step lie together.
 *
 * Measured (one B200, us per launch back to back, interpreter -> here): silu(x) * y of 24 000 500 f16 values 59.1 -> 28.8 (5.0 TB/s; 90
 * warp instructions per 128 values, issue slots 0.58 busy), f32 57.6 -> 47.3 (6.1 TB/s); x + y in f32 of 10^6 7.7 -> 4.2, 10^7 25.0 -> 21.2,
 * 40 000 003 76.8 -> 75.6, 8 * 10^7 149.0 -> 146.5 (6.55 TB/s, the rate of a copy); f16 of 24 000 500 34.6 -> 25.8. Eight groups per
 * thread and operand in f32: four keep more warps and pages open and were slower (8 * 10^7 154); SiLU of 2-byte elements is bound by issue
 * as well, and keeps twice the warps with two.
 */
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "gint_form_types.h"
#include "gint_silu.cuh"

namespace gint {

enum { FLAT_F32 = 0, FLAT_F16, FLAT_BF16 };
template <int TYPE> __host__ __device__ constexpr int flat_elements() { return TYPE == FLAT_F32 ? 4 : 8; }   // of a group: 16 bytes

template <int TYPE, int E> __device__ __forceinline__ void flat_values(const uint4 &g, float (&v)[E])
{
    const uint32_t w[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
    for (int i = 0; i < E; i++) {
        if constexpr (TYPE == FLAT_F32) v[i] = __uint_as_float(w[i]);
        else if constexpr (TYPE == FLAT_F16) v[i] = __half2float(__ushort_as_half((unsigned short)(w[i / 2] >> (16 * (i & 1)))));
        else v[i] = __uint_as_float(i & 1 ? w[i / 2] & 0xFFFF0000u : w[i / 2] << 16);
    }
}
template <int TYPE, int E> __device__ __forceinline__ uint4 flat_group(const float (&v)[E])
{
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if constexpr (TYPE == FLAT_F32) w[i] = __float_as_uint(v[i]);
        else if constexpr (TYPE == FLAT_F16) asm("cvt.rn.f16x2.f32 %0, %2, %1;" : "=r"(w[i]) : "f"(v[2 * i]), "f"(v[2 * i + 1]));
        else asm("cvt.rn.bf16x2.f32 %0, %2, %1;" : "=r"(w[i]) : "f"(v[2 * i]), "f"(v[2 * i + 1]));
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}
template <int TYPE, int MAP> __device__ __forceinline__ uint4 flat_map(const FlatArgs &a, const uint4 &x, const uint4 &y)
{
    constexpr int E = flat_elements<TYPE>();
    float v[E];
    flat_values<TYPE, E>(x, v);
    if (MAP & FLAT_SILU) silu(v, a.silu);
    if (MAP & (FLAT_ADD | FLAT_MUL)) {
        float w[E];
        flat_values<TYPE, E>(y, w);
#pragma unroll
        for (int i = 0; i < E; i++) v[i] = MAP & FLAT_ADD ? __fadd_rn(w[i], v[i]) : __fmul_rn(w[i], v[i]);
    }
    return flat_group<TYPE, E>(v);
}
template <int TYPE> __device__ __forceinline__ float flat_value(const void *base, u64 i)
{
    if constexpr (TYPE == FLAT_F32) return reinterpret_cast<const float *>(base)[i];
    else if constexpr (TYPE == FLAT_F16) return __half2float(reinterpret_cast<const __half *>(base)[i]);
    else return __bfloat162float(reinterpret_cast<const __nv_bfloat16 *>(base)[i]);
}

template <int TYPE, int MAP> __device__ __forceinline__ void flat_loop(const FlatArgs &a)
{
    constexpr int U = TYPE == FLAT_F32 ? 8 : MAP & FLAT_SILU ? 2 : 4;   // groups on their way per thread
    const uint32_t threads = gridDim.x * blockDim.x, me = blockIdx.x * blockDim.x + threadIdx.x;
    const uint4 *const x = reinterpret_cast<const uint4 *>(a.x), *const y = reinterpret_cast<const uint4 *>(a.y);
    uint4 *const z = reinterpret_cast<uint4 *>(a.z);
    /* a warp takes 32 U groups that lie together at a time */
    const bool few = a.end - a.begin <= threads;   // (a group per thread)
    uint32_t g = a.begin + (few ? me : (me >> 5) * (32u * U) + (me & 31u));
    uint4 gx[U], gy[U];
    for (; g < a.end; g += threads * U) {
        if (!few && g + 32u * (U - 1) < a.end) {
#pragma unroll
            for (int k = 0; k < U; k++) {
                gx[k] = x[g + 32u * k];
                if (MAP & (FLAT_ADD | FLAT_MUL)) gy[k] = y[g + 32u * k];
            }
#pragma unroll
            for (int k = 0; k < U; k++) z[g + 32u * k] = flat_map<TYPE, MAP>(a, gx[k], gy[k]);
        } else {
            for (uint32_t k = g; k < a.end; k += few ? threads : 32u) {
                gx[0] = x[k];
                if (MAP & (FLAT_ADD | FLAT_MUL)) gy[0] = y[k];
                z[k] = flat_map<TYPE, MAP>(a, gx[0], gy[0]);
            }
        }
    }
    if (me < a.rest) {   // the elements behind the last group, one per thread
        const u64 i = (u64)flat_elements<TYPE>() * a.end + me;
        float r[2] = {flat_value<TYPE>(a.x, i), 1.0f};
        if (MAP & FLAT_SILU) silu(r, a.silu);
        if (MAP & FLAT_ADD) r[0] = __fadd_rn(flat_value<TYPE>(a.y, i), r[0]);
        if (MAP & FLAT_MUL) r[0] = __fmul_rn(flat_value<TYPE>(a.y, i), r[0]);
        if constexpr (TYPE == FLAT_F32) reinterpret_cast<float *>(a.z)[i] = r[0];
        else if constexpr (TYPE == FLAT_F16) reinterpret_cast<__half *>(a.z)[i] = __float2half_rn(r[0]);
        else reinterpret_cast<__nv_bfloat16 *>(a.z)[i] = __float2bfloat16_rn(r[0]);
    }
}

template <int TYPE> __device__ __forceinline__ void flat_body(const FlatArgs &a)
{
    switch (a.map) {
    case FLAT_ADD: flat_loop<TYPE, FLAT_ADD>(a); break;
    case FLAT_MUL: flat_loop<TYPE, FLAT_MUL>(a); break;
    case FLAT_SILU: flat_loop<TYPE, FLAT_SILU>(a); break;
    case FLAT_SILU | FLAT_ADD: flat_loop<TYPE, FLAT_SILU | FLAT_ADD>(a); break;
    case FLAT_SILU | FLAT_MUL: flat_loop<TYPE, FLAT_SILU | FLAT_MUL>(a); break;
    }
}

}  // namespace gint

#define GINT_DEFINE_FLAT_KERNEL(name, type) \
    extern "C" __global__ void __launch_bounds__(256, gint::type == gint::FLAT_F32 ? 2 : 4) gint_form_flat_##name(const __grid_constant__ gint::FlatArgs a) { gint::flat_body<gint::type>(a); }
