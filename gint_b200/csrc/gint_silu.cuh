/*
 * gint_silu.cuh -- x / (exp(-x) + c) for several values at once, the quotient correctly rounded as by __fdiv_rn.
 *
 * A division per element costs its steps, a test of the operands' exponents and a branch around the general case, which also keeps
 * the elements of a group apart. For c = 1 the divisor is at least 1, and the quotient alone tells whether the plain steps hold:
 * reciprocal, one Newton step, then two corrections of the quotient by its exact remainder (P. Markstein, Computation of Elementary
 * Functions on the IBM RISC System/6000 Processor, 1990), in packed pairs. With d >= 1 and 2^-100 <= |q| <= 2^100 every remainder
 * x - d q is exact (its last bit is at least 2^-23 * 2^-124) and no step over- or underflows; if one of the group's quotients lies outside
 * (zeros, infinities, NaN, exp(-x) near overflow), the group takes the general division. Measured: silu(rmsnorm) + residual over 65536
 * rows of 1024 155 -> 137 us.
 */
#pragma once

#include <cuda_runtime.h>

namespace gint {

typedef unsigned long long u64;

__device__ __forceinline__ u64 pair(float x, float y) { u64 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y)); return r; }
__device__ __forceinline__ void unpair(u64 v, float &x, float &y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ u64 pair_fma(u64 x, u64 y, u64 z) { u64 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z)); return r; }
__device__ __forceinline__ u64 pair_mul(u64 x, u64 y) { u64 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y)); return r; }

template <int N> __device__ __forceinline__ void silu(float (&x)[N], float c)
{
    static_assert(N % 2 == 0, "pairs");
    float minus_d[N], q[N];
    float lo = 1.0f, hi = 1.0f;
#pragma unroll
    for (int i = 0; i < N; i++) minus_d[i] = __fsub_rn(-c, expf(-x[i]));
    const u64 one = pair(1.0f, 1.0f);
#pragma unroll
    for (int i = 0; i < N; i += 2) {
        float r0, r1;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(-minus_d[i]));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(-minus_d[i + 1]));
        const u64 n = pair(minus_d[i], minus_d[i + 1]), v = pair(x[i], x[i + 1]);
        u64 y = pair(r0, r1);
        y = pair_fma(y, pair_fma(n, y, one), y);
        u64 t = pair_mul(v, y);
        t = pair_fma(pair_fma(n, t, v), y, t);
        t = pair_fma(pair_fma(n, t, v), y, t);
        unpair(t, q[i], q[i + 1]);
    }
#pragma unroll
    for (int i = 0; i < N; i++) {   // (a NaN must not get lost: min.NaN, max.NaN)
        asm("min.NaN.f32 %0, %1, %2;" : "=f"(lo) : "f"(lo), "f"(fabsf(q[i])));
        asm("max.NaN.f32 %0, %1, %2;" : "=f"(hi) : "f"(hi), "f"(fabsf(q[i])));
    }
    if (c == 1.0f && lo >= 0x1p-100f && hi <= 0x1p100f) {
#pragma unroll
        for (int i = 0; i < N; i++) x[i] = q[i];
    } else {
#pragma unroll
        for (int i = 0; i < N; i++) x[i] = __fdiv_rn(x[i], __fadd_rn(-minus_d[i], 0.0f));   // (exp(-x) + c is never -0, as -minus_d is where it is zero)
    }
}

}  // namespace gint
