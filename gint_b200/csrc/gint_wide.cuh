/*
 * gint_wide.cuh -- the streaming interpreter: programs whose tile loops the host has found again (gint_capi.cu: wide_transform)
 * run their loop bodies on U consecutive tiles at a time.
 *
 * A bytecode program is straight-line: a pass over a row of 4096 values is the same handful of instructions 32 times, with
 * the tile offset moved on. The tile kernels (gint_interp.cuh) execute them one tile at a time, and what bounds them is not
 * memory but issue: RMSNorm rows took 137 warp instructions per 128-value tile (two passes), a + b over a length that
 * fills no last tile 148, per-head bf16 RMSNorm 246 (ncu, smsp__inst_executed). Here the stream contains the body once, between
 * a LoopBegin and a LoopEnd, and every instruction of it is executed for U tiles by one dispatch: the fetch, the branch, the
 * descriptor reads and the bounds checks are paid once per U tiles, U tiles of every operand are in flight without any
 * staging, and nothing depends on the alignment of a row.
 *
 * State. A pool slot holds U tiles (named registers as in gint_interp.cuh with K = U). Inside a loop an instruction works on
 * all U tiles of its slots (its opcode is GINT_WIDE_FIRST + op); outside of loops on tile 0 alone, with the ordinary handlers.
 * LoopBegin copies what is on the stack to all U tiles. A running
 * sum is kept in tile 0 and takes the U tiles in order (AccAdd, AccFMA), so every sum has the terms and the order of the
 * program as written: results are bit-identical. The one exception are sums of 2-byte 2DT tiles in the vector layout, whose terms
 * are added in another order (wide_vector in gint_wide_host.h).
 *
 * One warp runs one logical program. Programs that are nothing but one loop over 1-D tiles, whose logical programs follow one
 * another in memory, run "flat": the whole launch is one loop, cut among all warps.
 *
 * Measured (one B200, us per launch on the device, tile kernels -> here): a + b over 40 000 003 elements 84 -> 76 (53 warp instructions
 * per tile; 6.2 TB/s per pass); a * sigmoid(a) * b in f16 over as many 133 -> 93 (162); RMSNorm of 10 000 unaligned rows of 2029 values
 * 72 -> 56 (113); RMSNorm of 50 000 bf16 rows of 128 23.4 -> 18.9 (166), of 512 82 -> 46. U = 8 with 3 slots (128 registers, 16 warps per SM) beats U = 8 with 2 slots (96
 * registers, 20 warps; f16 57 against 67: calls spill) and U = 4 with 4 slots for long loops (79 against 83; 59 against 64); short
 * loops leave U = 8 half empty (heads of 128: 150 at U = 4, 210 at U = 8). What bounds the flat programs is memory (a + b) and the
 * exponential and division (f16); the row programs wait for memory round trips and for the instruction cache.
 */
#pragma once

#include "gint_interp.cuh"

namespace gint {

/* wide form: an element-wise instruction or a tile access in a loop body. Of the math that the tile kernels run out of line only
 * division, square root and reciprocal, which take four values per call (div4 and the like below): 4 U calls per handler would make
 * every live pool register a saved one. */
template <int OP> __host__ __device__ constexpr bool wide_ok()
{
    if constexpr (OP >= GINT_N_OPCODES) return false;
    else return GINT_WIDE_OP(OP);
}
template <int OP> __host__ __device__ constexpr bool narrow_ok()
{
    if constexpr (OP >= GINT_N_OPCODES) return false;
    else return GINT_WIDE_NARROW_OP(OP);
}
template <int OP> struct LoopForm { static constexpr bool is = false; };
#define GINT_X_LOOP(name, num, expr_, lay, dt, d0, len, ...)                                                                 \
    template <> struct LoopForm<num> {                                                                                       \
        static constexpr bool is = true;                                                                                     \
        static constexpr int expr = expr_, layout = lay, dtype = dt, depth = d0;                                             \
    };
GINT_WIDE_LOOP_LIST(GINT_X_LOOP)
#undef GINT_X_LOOP
template <int OP, int SP, int P> __host__ __device__ constexpr bool wide_valid()
{
    if constexpr (LoopForm<OP>::is) return SP == LoopForm<OP>::depth && SP <= P;
    else if constexpr (OP >= GINT_WIDE_FIRST) {
        if constexpr (!wide_ok<OP - GINT_WIDE_FIRST>()) return false;
        else return op_valid<OP - GINT_WIDE_FIRST, SP, P, 1>();
    } else if constexpr (OP < GINT_N_OPCODES) {
        if constexpr (OP == OP_Halt) return SP <= P;
        else if constexpr (!narrow_ok<OP>()) return false;
#ifdef GINT_WIDE_V
        else if constexpr (MemOp<OP>::is) return false;   // (programs with tile accesses outside of loops keep the natural layout)
#endif
        else return op_valid<OP, SP, P, 1>();
    } else {
        if constexpr (OP == WOP_LoopBegin || OP == WOP_LoopEnd) return SP <= P;
        else if constexpr (OP == WOP_Square || OP == WOP_Silu || OP == WOP_Remap) return SP >= 1 && SP <= P;
        else if constexpr (OP == WOP_AccAdd || OP == WOP_MulKeep || OP == WOP_AccFMASquare) return SP >= 2 && SP <= P;
        else if constexpr (OP == WOP_AccFMA) return SP >= 3 && SP <= P;
        else return false;
    }
}
template <int OP> __host__ __device__ constexpr int wide_net()
{
    if constexpr (LoopForm<OP>::is) return 0;
    else if constexpr (OP >= GINT_WIDE_FIRST) return OpInfo<OP - GINT_WIDE_FIRST>::net_effect;
    else if constexpr (OP < GINT_N_OPCODES) return OpInfo<OP>::net_effect;
    else return OP == WOP_AccAdd || OP == WOP_AccFMASquare ? -1 : OP == WOP_AccFMA ? -2 : 0;
}

/* the loop's state: tile number of the first of the U tiles in progress, tiles left including them */
__device__ __forceinline__ void loop_state(int &chunk, int &left)
{
    asm volatile("mov.b32 %0, %%gchunk; mov.b32 %1, %%gleft;" : "=r"(chunk), "=r"(left));
}

/* One predicated access: element K of an operand's tiles if K < limit, else zero. In PTX because a branch around each of 4 U
 * accesses per handler makes a control-flow graph that the assembler takes minutes for. */
template <int DT, int K> __device__ __forceinline__ float load_below(const char *p, int limit)
{
    uint32_t x;
    if constexpr (DT == DT_F32)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %2, %3;\n\tmov.b32 %0, 0;\n\t@p ld.global.b32 %0, [%1];\n\t}" : "=r"(x) : "l"(p), "n"(K), "r"(limit) : "memory");
    else if constexpr (DT == DT_U8)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %2, %3;\n\tmov.b32 %0, 0;\n\t@p ld.global.u8 %0, [%1];\n\t}" : "=r"(x) : "l"(p), "n"(K), "r"(limit) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %2, %3;\n\tmov.b32 %0, 0;\n\t@p ld.global.u16 %0, [%1];\n\t}" : "=r"(x) : "l"(p), "n"(K), "r"(limit) : "memory");
    if constexpr (DT == DT_F32) return __uint_as_float(x);
    else if constexpr (DT == DT_F16) return __half2float(__ushort_as_half((unsigned short)x));
    else if constexpr (DT == DT_BF16) return __uint_as_float(x << 16);
    else return (float)x;
}
template <int DT, int K> __device__ __forceinline__ void store_below(char *p, float v, int limit)
{
    if constexpr (DT == DT_F32)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %2, %3;\n\t@p st.global.b32 [%1], %0;\n\t}" ::"f"(v), "l"(p), "n"(K), "r"(limit) : "memory");
    else if constexpr (DT != DT_U8) {
        const unsigned short h = DT == DT_F16 ? __half_as_ushort(__float2half_rn(v)) : __bfloat16_as_ushort(__float2bfloat16_rn(v));
        asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %2, %3;\n\t@p st.global.b16 [%1], %0;\n\t}" ::"h"(h), "l"(p), "n"(K), "r"(limit) : "memory");
    }
}
#ifdef GINT_WIDE_V
/* four consecutive elements, aligned to their size */
template <int DT, bool STORE> __device__ __forceinline__ void access_four(char *p, float &a, float &b, float &c, float &d)
{
    if constexpr (DT == DT_F32) {
        if constexpr (STORE) asm volatile("st.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
        else asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(a), "=f"(b), "=f"(c), "=f"(d) : "l"(p) : "memory");
    } else if constexpr (DT == DT_U8) {
        uint32_t x;
        asm volatile("ld.global.b32 %0, [%1];" : "=r"(x) : "l"(p) : "memory");
        a = (float)(x & 0xFFu); b = (float)((x >> 8) & 0xFFu); c = (float)((x >> 16) & 0xFFu); d = (float)(x >> 24);
    } else if constexpr (STORE) {
        uint32_t x, y;
        if constexpr (DT == DT_F16) {
            asm("cvt.rn.f16x2.f32 %0, %2, %1;" : "=r"(x) : "f"(a), "f"(b));
            asm("cvt.rn.f16x2.f32 %0, %2, %1;" : "=r"(y) : "f"(c), "f"(d));
        } else {
            asm("cvt.rn.bf16x2.f32 %0, %2, %1;" : "=r"(x) : "f"(a), "f"(b));
            asm("cvt.rn.bf16x2.f32 %0, %2, %1;" : "=r"(y) : "f"(c), "f"(d));
        }
        asm volatile("st.global.v2.b32 [%0], {%1, %2};" ::"l"(p), "r"(x), "r"(y) : "memory");
    } else {
        uint32_t x, y;
        asm volatile("ld.global.v2.b32 {%0, %1}, [%2];" : "=r"(x), "=r"(y) : "l"(p) : "memory");
        if constexpr (DT == DT_BF16) {
            a = __uint_as_float(x << 16); b = __uint_as_float(x & 0xFFFF0000u);
            c = __uint_as_float(y << 16); d = __uint_as_float(y & 0xFFFF0000u);
        } else {
            asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tcvt.f32.f16 %0, l;\n\tcvt.f32.f16 %1, h;\n\t}" : "=f"(a), "=f"(b) : "r"(x));
            asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\tcvt.f32.f16 %0, l;\n\tcvt.f32.f16 %1, h;\n\t}" : "=f"(c), "=f"(d) : "r"(y));
        }
    }
}
#endif
template <int DT, bool STORE, int K> __device__ __forceinline__ void access_below(char *p, float &v, int limit)
{
    if constexpr (STORE) store_below<DT, K>(p, v, limit);
    else v = load_below<DT, K>(p, limit);
}
template <int DT, int U, bool STORE, int... J>   // 1-D layout: element 32 J of tile J / 4, width value J % 4
__device__ __forceinline__ void masked_1d(char *p, long long step, int limit, float (&v)[U][4], std::integer_sequence<int, J...>)
{
    ((access_below<DT, STORE, J * 32>(p, v[J / 4][J % 4], limit), p += step), ...);
}
template <int DT, int U, bool STORE, int... J>   // 2DT layout: element 32 J of width value w
__device__ __forceinline__ void masked_2dt(char *p, long long step, int limit, float (&v)[U][4], int w, std::integer_sequence<int, J...>)
{
    ((access_below<DT, STORE, J * 32>(p, v[J][w], limit), p += step), ...);
}

#ifdef GINT_WIDE_V
/* 1-D: element 128 u + w behind the lane's first; 2DT: element 128 g + j behind the lane's first is tile 4 g + j */
template <int DT, int U, bool STORE, int... J>
__device__ __forceinline__ void masked_1d_v(char *p, int limit, float (&v)[U][4], std::integer_sequence<int, J...>)
{
    (access_below<DT, STORE, (J / 4) * 128 + J % 4>(p + ((J / 4) * 128 + J % 4) * ElemSize<DT>::value, v[J / 4][J % 4], limit), ...);
}
template <int DT, int U, bool STORE, int... J>
__device__ __forceinline__ void masked_2dt_v(char *p, int limit, float (&v)[U][4], int w, std::integer_sequence<int, J...>)
{
    (access_below<DT, STORE, (J / 4) * 128 + J % 4>(p + ((J / 4) * 128 + J % 4) * ElemSize<DT>::value, v[J][w], limit), ...);
}

/* U tiles of one operand in the vector layout. The lane's values are four consecutive elements instead of four that lie 32 apart:
 * of a 1-D tile elements 4 l .. 4 l + 3 (width values 0 .. 3), of four 2DT tiles side by side (128 elements of dimension 1) elements
 * 4 l .. 4 l + 3 (tiles 0 .. 3), one access of 4 to 16 bytes instead of four. The host has proved stride 1 along dimension 1 and the
 * alignment of every such group, and that nothing in the program can tell the layouts apart (wide_vector in gint_wide_host.h). */
template <int LAYOUT, int DT, int U, bool STORE>
__device__ __forceinline__ void wide_rw(const TileInfo *ti, uint32_t operand, int lane, int chunk, int left, float (&v)[U][4])
{
    constexpr int ESZ = ElemSize<DT>::value, STEP = LAYOUT == LAY_1D ? 128 : 32;
    const int arg = operand & 15;
    const int off = (int)(operand >> 4) + chunk * STEP;
    char *base = reinterpret_cast<char *>(ti->ptr[arg]);
    const int n1 = ti->s1[arg].x;
    const bool full = left >= U && off + U * STEP <= n1;
    const int limit = min(left * STEP, n1 - off) - 4 * lane;
    if constexpr (LAYOUT == LAY_1D) {
        char *p = base + (long long)(off + 4 * lane) * ESZ;
        if (full) {
#pragma unroll
            for (int u = 0; u < U; u++) access_four<DT, STORE>(p + u * 128 * ESZ, v[u][0], v[u][1], v[u][2], v[u][3]);
        } else {
            masked_1d_v<DT, U, STORE>(p, limit, v, std::make_integer_sequence<int, 4 * U>());
        }
    } else {
        const int2 s2 = ti->s2[arg];
        const int j0 = ti->adv[arg];
        if (full && j0 + 4 <= s2.x) {
#pragma unroll
            for (int w = 0; w < 4; w++) {
                char *p = base + (long long)(off + 4 * lane + (j0 + w) * s2.y) * ESZ;
#pragma unroll
                for (int g = 0; g < U; g += 4) access_four<DT, STORE>(p + g * 32 * ESZ, v[g][w], v[g + 1][w], v[g + 2][w], v[g + 3][w]);
            }
        } else {
#pragma unroll
            for (int w = 0; w < 4; w++)
                masked_2dt_v<DT, U, STORE>(base + (long long)(off + 4 * lane + (j0 + w) * s2.y) * ESZ, j0 + w < s2.x ? limit : INT32_MIN, v, w,
                                           std::make_integer_sequence<int, U>());
        }
    }
}
#else
/* U tiles of one operand. The tiles follow one another along dimension 1 (128 elements each in the 1-D layout, 32 in 2DT). All U
 * in range, dimension 1 with stride 1: 4 U accesses at immediate offsets from one or four pointers. Otherwise every access is
 * predicated and the pointer advances by the stride. (tile_rw computes every index in 32 bits; the host takes a program to these
 * kernels only where no index leaves 31 bits, so the addresses are the same.) */
template <int LAYOUT, int DT, int U, bool STORE>
__device__ __forceinline__ void wide_rw(const TileInfo *ti, uint32_t operand, int lane, int chunk, int left, float (&v)[U][4])
{
    constexpr int ESZ = ElemSize<DT>::value, STEP = LAYOUT == LAY_1D ? 128 : 32;
    const int arg = operand & 15;
    const int off = (int)(operand >> 4) + chunk * STEP;
    char *base = reinterpret_cast<char *>(ti->ptr[arg]);
    const int2 s1 = ti->s1[arg];
    const bool full = left >= U && off + U * STEP <= s1.x && s1.y == 1;
    if constexpr (LAYOUT == LAY_1D) {
        if (full) {
            char *p = base + (long long)(lane + off) * ESZ;
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int w = 0; w < 4; w++) {
                    if constexpr (STORE) store_elem<DT>(p + (u * 128 + w * 32) * ESZ, v[u][w]);
                    else v[u][w] = load_elem<DT>(p + (u * 128 + w * 32) * ESZ);
                }
            return;
        }
        const int limit = min(left * 128, s1.x - off) - lane;   // element k of the U tiles exists iff k < limit
        char *p = base + (long long)((lane + off) * s1.y) * ESZ;
        const long long step = (long long)s1.y * (32 * ESZ);
        masked_1d<DT, U, STORE>(p, step, limit, v, std::make_integer_sequence<int, 4 * U>());
    } else {
        const int2 s2 = ti->s2[arg];
        const int j0 = ti->adv[arg];
        if (full && j0 + 4 <= s2.x) {
#pragma unroll
            for (int w = 0; w < 4; w++) {
                char *p = base + (long long)(lane + off + (j0 + w) * s2.y) * ESZ;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    if constexpr (STORE) store_elem<DT>(p + u * 32 * ESZ, v[u][w]);
                    else v[u][w] = load_elem<DT>(p + u * 32 * ESZ);
                }
            }
            return;
        }
        const int limit = min(left * 32, s1.x - off) - lane;
        const long long step = (long long)s1.y * (32 * ESZ);
#pragma unroll
        for (int w = 0; w < 4; w++) {
            const int n = j0 + w < s2.x ? limit : INT32_MIN;
            char *p = base + (long long)((lane + off) * s1.y + (j0 + w) * s2.y) * ESZ;
            masked_2dt<DT, U, STORE>(p, step, n, v, w, std::make_integer_sequence<int, U>());
        }
    }
}

#endif

template <int U, int SLOT, int... KI> __device__ __forceinline__ void wide_read(float (&v)[U][4], std::integer_sequence<int, KI...>)
{
    (slot_read<U, SLOT, KI>(v[KI]), ...);
}
template <int U, int SLOT, int... KI> __device__ __forceinline__ void wide_write(const float (&v)[U][4], std::integer_sequence<int, KI...>)
{
    (slot_write<U, SLOT, KI>(v[KI]), ...);
}

/* tile 0 of slot `ACC` takes tile KI of the operands if the loop still has it */
template <int OP, int SP, int U, int KI> __device__ __forceinline__ void accumulate_one(int left)
{
    if (KI < left) {
        if constexpr (OP == WOP_AccAdd) {
            r_add2<gs<U>(SP - 2, 0, 0), gs<U>(SP - 1, KI, 0), gs<U>(SP - 2, 0, 0)>();
            r_add2<gs<U>(SP - 2, 0, 1), gs<U>(SP - 1, KI, 1), gs<U>(SP - 2, 0, 1)>();
        } else if constexpr (OP == WOP_AccFMASquare) {
            r_fma2<gs<U>(SP - 2, 0, 0), gs<U>(SP - 1, KI, 0), gs<U>(SP - 1, KI, 0), gs<U>(SP - 2, 0, 0)>();
            r_fma2<gs<U>(SP - 2, 0, 1), gs<U>(SP - 1, KI, 1), gs<U>(SP - 1, KI, 1), gs<U>(SP - 2, 0, 1)>();
        } else {
            r_fma2<gs<U>(SP - 3, 0, 0), gs<U>(SP - 1, KI, 0), gs<U>(SP - 2, KI, 0), gs<U>(SP - 3, 0, 0)>();
            r_fma2<gs<U>(SP - 3, 0, 1), gs<U>(SP - 1, KI, 1), gs<U>(SP - 2, KI, 1), gs<U>(SP - 3, 0, 1)>();
        }
    }
}

/* Division, square root, reciprocal and SiLU of four values, out of line: each has a slow path for operands near the ends of the
 * exponent range, and 4 U copies of it in every handler make a control-flow graph that the assembler takes minutes for. */
static __device__ __noinline__ float4 div4(float4 x, float4 y) { return make_float4(__fdiv_rn(x.x, y.x), __fdiv_rn(x.y, y.y), __fdiv_rn(x.z, y.z), __fdiv_rn(x.w, y.w)); }
static __device__ __noinline__ float4 sqrt4(float4 x) { return make_float4(__fsqrt_rn(x.x), __fsqrt_rn(x.y), __fsqrt_rn(x.z), __fsqrt_rn(x.w)); }
static __device__ __noinline__ float4 rcp4(float4 x) { return make_float4(__frcp_rn(x.x), __frcp_rn(x.y), __frcp_rn(x.z), __frcp_rn(x.w)); }
static __device__ __noinline__ float4 silu4(float4 x, float c)
{
    return make_float4(__fdiv_rn(x.x, __fadd_rn(expf(-x.x), c)), __fdiv_rn(x.y, __fadd_rn(expf(-x.y), c)),
                       __fdiv_rn(x.z, __fadd_rn(expf(-x.z), c)), __fdiv_rn(x.w, __fadd_rn(expf(-x.w), c)));
}
template <int OP> __host__ __device__ constexpr bool four_at_a_time()
{
    return OP == OP_FDiv || OP == OP_FRDiv || OP == OP_FSqrt || OP == OP_FRcp || OP == WOP_Silu;
}
template <int OP, int SP, int U, int KI> __device__ __forceinline__ void exec_four(uint32_t operand)
{
    float t[4];
    slot_read<U, SP - 1, KI>(t);
    const float4 x = make_float4(t[0], t[1], t[2], t[3]);
    float4 r;
    if constexpr (OP == OP_FDiv || OP == OP_FRDiv) {
        float q[4];
        slot_read<U, SP - 2, KI>(q);
        const float4 y = make_float4(q[0], q[1], q[2], q[3]);
        r = OP == OP_FDiv ? div4(x, y) : div4(y, x);
    } else if constexpr (OP == OP_FSqrt) r = sqrt4(x);
    else if constexpr (OP == OP_FRcp) r = rcp4(x);
    else r = silu4(x, __uint_as_float(operand));
    const float o[4] = {r.x, r.y, r.z, r.w};
    slot_write<U, (OP == OP_FDiv || OP == OP_FRDiv) ? SP - 2 : SP - 1, KI>(o);
}

template <int OP, int SP, int P, int U, int... KI>
__device__ __forceinline__ void wide_exec(const uint32_t operand, const Ctx &cx, std::integer_sequence<int, KI...> seq)
{
    if constexpr (OP >= GINT_WIDE_FIRST) {
        constexpr int BASE = OP - GINT_WIDE_FIRST;
        if constexpr (MemOp<BASE>::is) {
            float v[U][4];
            int chunk, left;
            loop_state(chunk, left);
            if constexpr (MemOp<BASE>::store) {
                wide_read<U, SP - 1>(v, seq);
                wide_rw<MemOp<BASE>::layout, MemOp<BASE>::dtype, U, true>(cx.tiles, operand, cx.lane, chunk, left, v);
            } else {
                wide_rw<MemOp<BASE>::layout, MemOp<BASE>::dtype, U, false>(cx.tiles, operand, cx.lane, chunk, left, v);
                wide_write<U, SP>(v, seq);
            }
        } else if constexpr (four_at_a_time<BASE>()) {
            (exec_four<BASE, SP, U, KI>(operand), ...);
        } else {
            (exec_tile<BASE, SP, P, U, KI>(operand, cx), ...);
        }
    } else if constexpr (four_at_a_time<OP>() && OP < GINT_N_OPCODES) {
        exec_four<OP, SP, U, 0>(operand);
    } else if constexpr (OP == WOP_Remap) {
#ifdef GINT_WIDE_V
        const uint32_t area = block_scalar(0) + warp_here() * 512u;   // the warp's exchange area
        put_vector<U, SP - 1, 0>(area + (uint32_t)cx.lane * 16u);
        __syncwarp();
        take_natural<U, SP - 1, 0>(area + (uint32_t)cx.lane * 4u);
        __syncwarp();
#endif
#ifndef GINT_WIDE_V
    } else if constexpr (OP < GINT_N_OPCODES && GINT_WIDE_TILE_OP(OP)) {
        float v[1][4];
        if constexpr (MemOp<OP>::store) {
            slot_read<U, SP - 1, 0>(v[0]);
            wide_rw<MemOp<OP>::layout, MemOp<OP>::dtype, 1, true>(cx.tiles, operand, cx.lane, 0, 1, v);
        } else {
            wide_rw<MemOp<OP>::layout, MemOp<OP>::dtype, 1, false>(cx.tiles, operand, cx.lane, 0, 1, v);
            slot_write<U, SP, 0>(v[0]);
        }
#endif
    } else if constexpr (OP < GINT_N_OPCODES) {
        exec_tile<OP, SP, P, U, 0>(operand, cx);
    } else if constexpr (OP == WOP_AccAdd || OP == WOP_AccFMA || OP == WOP_AccFMASquare) {
        int chunk, left;
        loop_state(chunk, left);
        (accumulate_one<OP, SP, U, KI>(left), ...);
    } else if constexpr (OP == WOP_Square) {        // Dup, FMul
        (r_mul2<gs<U>(SP - 1, KI, 0), gs<U>(SP - 1, KI, 0), gs<U>(SP - 1, KI, 0)>(), ...);
        (r_mul2<gs<U>(SP - 1, KI, 1), gs<U>(SP - 1, KI, 1), gs<U>(SP - 1, KI, 1)>(), ...);
    } else if constexpr (OP == WOP_MulKeep) {       // [s, x] -> [s, s * x]
        (r_mul2<gs<U>(SP - 1, KI, 0), gs<U>(SP - 2, KI, 0), gs<U>(SP - 1, KI, 0)>(), ...);
        (r_mul2<gs<U>(SP - 1, KI, 1), gs<U>(SP - 2, KI, 1), gs<U>(SP - 1, KI, 1)>(), ...);
    } else if constexpr (OP == WOP_Silu) {          // Dup, FNeg, FExp, FAddImm c, FRDiv: x / (exp(-x) + c)
        (exec_four<WOP_Silu, SP, U, KI>(operand), ...);
    }
}

/* N operands of a whole-loop instruction (operand 0: the number of tiles); the last entry carries the next opcode */
template <int N, int J = 1> __device__ __forceinline__ void loop_operands(uint32_t (&ops)[N], uint32_t &opc, uint32_t at)
{
    if constexpr (J == N - 1) asm volatile("ld.shared.v2.u32 {%0, %1}, [%2+%3];" : "=r"(ops[J]), "=r"(opc) : "r"(at), "n"(8 * (J - 1)));
    else {
        asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(ops[J]) : "r"(at), "n"(8 * (J - 1)));
        loop_operands<N, J + 1>(ops, opc, at);
    }
}

/* A whole loop: iterations of U tiles, body values in local registers, the loads of an iteration in front. The same operations in
 * the same order on every element as the interpreted body (scalar mul and add: the packed ones of one handler would be contracted,
 * see fma_barrier in gint_interp.cuh). */
template <int OP, int SP, int SLOT_TILES, int U> __device__ __forceinline__ void run_loop(const Ctx &cx, uint32_t &opc)
{
    using Form = LoopForm<OP>;
    constexpr int X = Form::expr, L = Form::layout, D = Form::dtype;
    constexpr int N = X <= LX_FMASQ ? 2 : 4;
    uint32_t ops[N], at;
    asm volatile("mov.b32 %0, %%ge0; mov.b32 %1, %%gc;" : "=r"(ops[0]), "=r"(at));
    loop_operands<N>(ops, opc, at);
    asm volatile("ld.shared.v2.u32 {%%ge0, %%ge1}, [%%gc+%0]; add.u32 %%gc, %%gc, %1;" ::"n"(8 * (N - 1)), "n"(8 * N) : "memory");
    int chunk, left;
    loop_state(chunk, left);
    if (ops[0] != 0u) { chunk = 0; left = (int)ops[0]; }
    float s[4];
    if constexpr (SP > 0) slot_read<SLOT_TILES, (SP > 0 ? SP - 1 : 0), 0>(s);
    do {
        float a[U][4];
        wide_rw<L, D, U, false>(cx.tiles, ops[1], cx.lane, chunk, left, a);
        if constexpr (X <= LX_FMASQ) {
#pragma unroll
            for (int u = 0; u < U; u++)
                if (u < left) {
#pragma unroll
                    for (int w = 0; w < 4; w++)
                        s[w] = X == LX_SUM ? __fadd_rn(a[u][w], s[w]) : X == LX_SUMSQ ? __fadd_rn(__fmul_rn(a[u][w], a[u][w]), s[w]) : __fmaf_rn(a[u][w], a[u][w], s[w]);
                }
        } else {
            float b[U][4];
            wide_rw<L, D, U, false>(cx.tiles, ops[2], cx.lane, chunk, left, b);
#pragma unroll
                for (int u = 0; u < U; u++)
#pragma unroll
                    for (int w = 0; w < 4; w++) a[u][w] = __fmul_rn(b[u][w], __fmul_rn(s[w], a[u][w]));
            wide_rw<L, D, U, true>(cx.tiles, ops[N - 1], cx.lane, chunk, left, a);
        }
        chunk += U;
        left -= U;
    } while (left > 0);
    if constexpr (X <= LX_FMASQ) slot_write<SLOT_TILES, SP - 1, 0>(s);
}

/* LoopBegin: tiles 1 .. U - 1 of what is on the stack get the value of tile 0. Those of the free slots get zero, which no
 * instruction reads, but which tells the assembler that outside of loops only tile 0 of a slot is live: the whole-loop handlers have
 * the other registers to themselves. */
template <int SP, int U, int I> __device__ __forceinline__ void spread_one()
{
    constexpr int slot = I / (U - 1), tile = I % (U - 1) + 1;
    if constexpr (slot < SP) {
        r_mov<gs<U>(slot, tile, 0), gs<U>(slot, 0, 0)>();
        r_mov<gs<U>(slot, tile, 1), gs<U>(slot, 0, 1)>();
    } else {
        r_set64<gs<U>(slot, tile, 0)>(0ull);
        r_set64<gs<U>(slot, tile, 1)>(0ull);
    }
}
template <int SP, int U, int... I> __device__ __forceinline__ void spread_slots(std::integer_sequence<int, I...>)
{
    (spread_one<SP, U, I>(), ...);
}

template <int OP, int SP, int P, int U> __device__ __forceinline__ void wide_handler()
{
    constexpr int next_depth = SP + wide_net<OP>();
    uint32_t operand, opc;
    if constexpr (LoopForm<OP>::is) {
        const Ctx cx = handler_context();
        run_loop<OP, SP, U, (LoopForm<OP>::expr <= LX_FMASQ ? U : 4)>(cx, opc);
    } else if constexpr (OP == WOP_LoopEnd) {
        /* operand unused. Next U tiles: back to the body's first instruction, whose entries start at %gloop - 16 */
        int left;
        asm volatile("sub.s32 %%gleft, %%gleft, %1; add.s32 %%gchunk, %%gchunk, %1; mov.b32 %0, %%gleft;" : "=r"(left) : "n"(U));
        if (left > 0) {
            asm volatile("ld.shared.u32 %0, [%%gloop+-12]; ld.shared.v2.u32 {%%ge0, %%ge1}, [%%gloop+-8]; mov.b32 %%gc, %%gloop;" : "=r"(opc) :: "memory");
            asm volatile("brx.idx.uni %0, GTW%1; // %2 %3" ::"r"(opc), "n"(SP), "n"(SP), "n"(OP) : "memory");
        }
        state_advance(operand, opc);
    } else {
        const Ctx cx = handler_context();
        state_advance(operand, opc);
        if constexpr (OP == WOP_LoopBegin) {
            /* operand: number of tiles. A flat launch has set %gchunk and %gleft itself (operand 0). */
            asm volatile("mov.b32 %%gloop, %%gc; // %0" ::"n"(0));
            spread_slots<SP, U>(std::make_integer_sequence<int, P * (U - 1)>());
            if (operand != 0u) asm volatile("mov.b32 %%gchunk, 0; mov.b32 %%gleft, %0;" ::"r"(operand));
        } else {
            wide_exec<OP, SP, P, U>(operand, cx, std::make_integer_sequence<int, U>());
        }
    }
    if constexpr (!LoopForm<OP>::is && OP >= GINT_N_OPCODES && OP != WOP_LoopEnd && OP != WOP_Remap)
        asm volatile("brx.idx.uni %0, GTW%1; // %2 %3" ::"r"(opc), "n"(next_depth), "n"(SP), "n"(OP) : "memory");
    else
        asm volatile("brx.idx.uni %0, GTN%1; // %2 %3" ::"r"(opc), "n"(next_depth), "n"(SP), "n"(OP) : "memory");
}

template <int P, int KEY> __device__ __forceinline__ void wide_missing_label()
{
    constexpr int sp = KEY / GINT_N_TABLE, num = KEY % GINT_N_TABLE;
    if constexpr (!wide_valid<num, sp, P>()) asm volatile("GL%0_%1:" ::"n"(sp), "n"(num) : "memory");
}
template <int P, int... KEY> __device__ __forceinline__ void wide_missing_labels(std::integer_sequence<int, KEY...>)
{
    (wide_missing_label<P, KEY>(), ...);
}

/* The dispatch is that of gint_interp.cuh: interpret (labels, one table per depth, a switch only for reachability). */
template <int P, int U> __device__ __forceinline__ void wide_interpret(uint32_t code)
{
    asm volatile("ld.shared.u32 %%gkey, [%0+4]; ld.shared.v2.u32 {%%ge0, %%ge1}, [%0+8]; add.u32 %%gc, %0, 16;" ::"r"(code) : "memory");
    asm volatile(GINT_WIDE_BRANCH_TABLES "// %0" ::"n"(0));
    for (;;) {
        uint32_t key;
        asm volatile("mov.b32 %0, %%gkey;\n\tbrx.idx.uni %%gkey, GTN0;" : "=r"(key) :: "memory");
        switch (key) {
#define GINT_WCASE(num, spv)                                                                    \
    case (spv) * GINT_N_TABLE + (num):                                                           \
        if constexpr (wide_valid<num, spv, P>()) {                                               \
            asm volatile("GL%0_%1:" ::"n"(spv), "n"(num) : "memory");                            \
            if constexpr ((num) == OP_Halt) return;                                             \
            else wide_handler<num, spv, P, U>();                                                \
        }                                                                                       \
        continue;
#define GINT_WCASES(num) GINT_WCASE(num, 0) GINT_WCASE(num, 1) GINT_WCASE(num, 2) GINT_WCASE(num, 3) GINT_WCASE(num, 4)
#define GINT_WCASE_WIDE(num, spv)                                                                \
    case GINT_N_KEYS + (spv) * GINT_N_TABLE + (num):                                              \
        if constexpr ((num) != OP_Halt && wide_valid<GINT_WIDE_FIRST + num, spv, P>()) {          \
            asm volatile("GL%0_%1:" ::"n"(spv), "n"(GINT_WIDE_FIRST + num) : "memory");           \
            wide_handler<GINT_WIDE_FIRST + num, spv, P, U>();                                    \
        }                                                                                       \
        continue;
#define GINT_WCASES_WIDE(num) GINT_WCASE_WIDE(num, 0) GINT_WCASE_WIDE(num, 1) GINT_WCASE_WIDE(num, 2) GINT_WCASE_WIDE(num, 3) GINT_WCASE_WIDE(num, 4)
#define GINT_X_WOWN(name, num) GINT_WCASES(num)
#define GINT_X_LOOP(name, num, ...) GINT_WCASES(num)
#define GINT_X_WIDE(name, num, md, net) GINT_WCASES_WIDE(num)
#define GINT_X_NARROW(name, num, md, net) GINT_WCASES(num)
            GINT_WIDE_LOOP_LIST(GINT_X_LOOP)
            GINT_WIDE_OWN_LIST(GINT_X_WOWN)
            GINT_OPCODE_LIST(GINT_X_WIDE)
            GINT_OPCODE_LIST(GINT_X_NARROW)
#undef GINT_X_NARROW
#undef GINT_X_WIDE
#undef GINT_X_LOOP
#undef GINT_X_WOWN
#undef GINT_WCASES
#undef GINT_WCASES_WIDE
#undef GINT_WCASE_WIDE
#undef GINT_WCASE
        default:
            wide_missing_labels<P>(std::make_integer_sequence<int, 5 * GINT_N_TABLE>());
            return;
        }
    }
}

/* Shared memory: [program | descriptor block | one TileInfo per warp | vector layout: 512 bytes of exchange area per warp]. blockDim.x / 32 warps per block (launches of few logical
 * programs use blocks of one warp, so that every program gets an SM to itself). */
template <int P, int U> __device__ __forceinline__ void geval_wide_body(const LaunchArgs &a)
{
    pool_declare<P, U>();
    state_declare();
    asm volatile(".reg .b32 %%gloop; .reg .b32 %%gchunk; .reg .b32 %%gleft; // %0" ::"n"(0));
    uint2 *code_s = reinterpret_cast<uint2 *>(g_smem);
    gint_tensor_info *ti_s = reinterpret_cast<gint_tensor_info *>(g_smem + a.code_smem_bytes);
    TileInfo *tiles_s = reinterpret_cast<TileInfo *>(g_smem + a.code_smem_bytes + kTensorInfoSmemBytes);
    for (uint32_t i = threadIdx.x; i < a.n_slots; i += blockDim.x) code_s[i] = a.code ? a.code[i] : a.inline_code[i];
    {
        const int *src = reinterpret_cast<const int *>(&a.ti);
        int *dst = reinterpret_cast<int *>(ti_s);
        for (uint32_t i = threadIdx.x; i < sizeof(gint_tensor_info) / 4; i += blockDim.x) dst[i] = src[i];
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t warps = blockDim.x >> 5;
#ifdef GINT_WIDE_V
    if (threadIdx.x == 0) g_block[0] = (uint32_t)__cvta_generic_to_shared(tiles_s + warps);
#endif
    __syncthreads();
    Ctx cx{};
    cx.tiles = tiles_s + warp;
    cx.lane = lane;
    context_set(cx);
    const uint32_t code = (uint32_t)__cvta_generic_to_shared(code_s);
    const bool flat = a.flat_tiles != 0;
    /* flat: tiles [first, end) x flat_tiles, U at a time, with the descriptors of logical program 0; else one logical program per step */
    const uint32_t tiles = flat ? (a.end - a.first) * a.flat_tiles : 0u;
    const uint32_t n_groups = flat ? (tiles + (uint32_t)U - 1u) / (uint32_t)U : a.end - a.first;
    if (flat) decode_tiles<1>(ti_s, (int)a.n_tensors, 0u, 1u, cx.tiles, lane);
    pool_clear<2 * P * U>();
    for (uint32_t g = blockIdx.x * warps + warp; g < n_groups; g += gridDim.x * warps) {
        if (flat) {
            asm volatile("mov.b32 %%gchunk, %0; mov.b32 %%gleft, %1;" ::"r"(a.first * a.flat_tiles + g * (uint32_t)U), "r"(min(tiles - g * (uint32_t)U, (uint32_t)U)));
        } else {
            __syncwarp();  // every lane is done with the previous program's tile descriptors
            decode_tiles<1>(ti_s, (int)a.n_tensors, a.first + g, a.end, cx.tiles, lane, a.gather_mask, a.gather_index, a.gather_rows);
            if (a.prefetch_mask) prefetch_footprints<1>(a, cx.tiles, lane);
        }
        wide_interpret<P, U>(code);
    }
}

}  // namespace gint

#ifdef GINT_WIDE_V
#define GINT_WIDE_NAME(P, U) gint_geval_widev_##P##_##U
#else
#define GINT_WIDE_NAME(P, U) gint_geval_wide_##P##_##U
#endif
#define GINT_DEFINE_WIDE_KERNEL(P, U, BLOCKS)                                                                   \
    extern "C" __global__ void __launch_bounds__(gint::kThreadsPerBlock, BLOCKS)                                 \
        GINT_WIDE_NAME(P, U)(const __grid_constant__ gint::LaunchArgs a)                                    \
    {                                                                                                           \
        gint::geval_wide_body<P, U>(a);                                                                         \
    }
