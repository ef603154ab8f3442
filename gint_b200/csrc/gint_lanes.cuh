/*
 * gint_lanes.cuh -- small-matrix programs, compiled ahead of time.
 *
 * In a program of 2DW rows a lane owns a matrix (32 rows of 16 floats per logical program) and no instruction looks at another
 * lane. Interpreted, such programs are bound by issue and by what stands for registers: the batched 4x4 product took 20 dispatches
 * per two tiles, the 4x4 inverse 43 and 72 accesses to virtual registers in shared memory (12.7 M wavefronts per million
 * matrices), which is 1.4 and 3.6 times the time of their bytes. The streams of the two library programs do not depend on the batch, so the
 * kernels here hold them as straight code: instruction by instruction what the interpreter does, at compile time (gint_lane_programs.h
 * is written by the build from the recorded streams), with every stack entry and virtual register in hardware registers; lane permutations
 * and shuffles are renamings. A program whose instructions are not those of a recorded one is interpreted.
 *
 * One warp runs a tile at a time. The tiles to come are brought into a ring of stages in shared memory by coalesced 16-byte
 * asynchronous copies, 16 bytes of a row at a position that keeps the lanes' 16-byte reads free of bank conflicts; results leave the same way
 * through a tile of shared memory, so that global memory sees whole lines only.
 *
 * Measured (one B200, us, interpreter -> here; bound by memory now): inverse of 4 194 304 matrices 299 -> 89 (6.0 TB/s),
 * 1 048 576 89 -> 25, 33 24 -> 6; product of 4 194 304 174 -> 122 (6.6 TB/s, the rate of a copy), 1 048 576 54 -> 35, 33 21 -> 6.5.
 */
#pragma once

#include <cuda_runtime.h>

#include "gint_form_types.h"
#include "gint_lane_programs.h"
#include "gint_opcodes.h"

namespace gint {

extern __shared__ __align__(128) char g_form_smem[];

/* What is known of a program at compile time: which slots it loads and stores, in order of their numbers. */
template <class P> struct LaneProgram {
    __host__ __device__ static constexpr bool load(int i) { return P::code[i][0] == OP_LoadGlobal2DWF32; }
    __host__ __device__ static constexpr bool store(int i) { return P::code[i][0] == OP_StoreGlobal2DWF32; }
    __host__ __device__ static constexpr uint32_t mask(bool stores)
    {
        uint32_t m = 0;
        for (int i = 0; i < P::n; i++)
            if (stores ? store(i) : load(i)) m |= 1u << (P::code[i][1] & 15);
        return m;
    }
    static constexpr uint32_t loads = mask(false), stores = mask(true);
    __host__ __device__ static constexpr int count(uint32_t m) { int c = 0; for (; m; m &= m - 1) c++; return c; }
    __host__ __device__ static constexpr int index(uint32_t m, int t) { return count(m & ((1u << t) - 1u)); }
    __host__ __device__ static constexpr int slot(uint32_t m, int k) { int t = 0; for (;; t++) if ((m >> t) & 1u && k-- == 0) return t; }
    static constexpr int n_in = count(loads), n_out = count(stores);
};

/* position (16-byte groups) of group c of row m in a staged tile: the eight lanes of a wavefront hit eight bank groups */
__device__ __forceinline__ int lane_position(int m, int c) { return m * 4 + (c ^ ((m >> 1) & 3)); }

template <class P> struct LaneState {
    float stack[9][4], reg[8][4];
    float in[LaneProgram<P>::n_in][4][4], out[LaneProgram<P>::n_out][4][4];
};

/* instruction I at stack depth SP, then the rest (exec_tile in gint_interp.cuh gives the semantics) */
template <class P, int I, int SP> __device__ __forceinline__ void lane_run(LaneState<P> &s)
{
    using L = LaneProgram<P>;
    constexpr int op = P::code[I][0], T = SP - 1, S = SP - 2;
    constexpr uint32_t arg = (uint32_t)P::code[I][1];
    constexpr uint32_t sel[4] = {arg & 3u, (arg >> 8) & 3u, (arg >> 16) & 3u, (arg >> 24) & 3u};
    if constexpr (op == OP_Halt) return;
    else {
        constexpr bool push = op == OP_LoadGlobal2DWF32 || op == OP_LoadImm4F || op == OP_Dup || op == OP_DupBroadcastW || (op >= OP_FLoadReg0 && op <= OP_FLoadReg7);
        constexpr bool pop = op == OP_StoreGlobal2DWF32 || op == OP_Pop || op == OP_FAdd || op == OP_FMul || op == OP_FSub || op == OP_FRSub || op == OP_FDiv ||
                             op == OP_FShuf2 || (op >= OP_FStoreReg0 && op <= OP_FStoreReg7);
        constexpr int next = SP + (push ? 1 : 0) - (pop ? 1 : 0) + (op == OP_Dup2 ? 2 : 0);
        static_assert(push || pop || op == OP_Dup2 || op == OP_Swap || op == OP_FPermW, "not a lane program");
        float t[4] = {}, b[4] = {};
        if constexpr (SP >= 1) {
#pragma unroll
            for (int w = 0; w < 4; w++) t[w] = s.stack[SP >= 1 ? T : 0][w];
        }
        if constexpr (SP >= 2) {
#pragma unroll
            for (int w = 0; w < 4; w++) b[w] = s.stack[SP >= 2 ? S : 0][w];
        }
#pragma unroll
        for (int w = 0; w < 4; w++) {
            if constexpr (op == OP_LoadGlobal2DWF32) s.stack[SP][w] = s.in[L::index(L::loads, (int)(arg & 15u))][arg >> 6][w];
            else if constexpr (op == OP_StoreGlobal2DWF32) s.out[L::index(L::stores, (int)(arg & 15u))][arg >> 6][w] = t[w];
            else if constexpr (op == OP_LoadImm4F) s.stack[SP][w] = (float)(signed char)(arg >> (8 * w));
            else if constexpr (op == OP_Dup) s.stack[SP][w] = t[w];
            else if constexpr (op == OP_Dup2) { s.stack[SP][w] = b[w]; s.stack[SP + 1][w] = t[w]; }
            else if constexpr (op == OP_Swap) { s.stack[T][w] = b[w]; s.stack[S][w] = t[w]; }
            else if constexpr (op == OP_DupBroadcastW) s.stack[SP][w] = t[arg];
            else if constexpr (op == OP_FPermW) s.stack[T][w] = t[sel[w]];
            else if constexpr (op == OP_FShuf2) s.stack[S][w] = w < 2 ? b[sel[w]] : t[sel[w]];
            else if constexpr (op >= OP_FLoadReg0 && op <= OP_FLoadReg7) s.stack[SP][w] = s.reg[op - OP_FLoadReg0][w];
            else if constexpr (op >= OP_FStoreReg0 && op <= OP_FStoreReg7) s.reg[op - OP_FStoreReg0][w] = t[w];
            else if constexpr (op == OP_FAdd) s.stack[S][w] = __fadd_rn(t[w], b[w]);
            else if constexpr (op == OP_FMul) s.stack[S][w] = __fmul_rn(t[w], b[w]);
            else if constexpr (op == OP_FSub) s.stack[S][w] = __fsub_rn(t[w], b[w]);
            else if constexpr (op == OP_FRSub) s.stack[S][w] = __fsub_rn(b[w], t[w]);
            else if constexpr (op == OP_FDiv) s.stack[S][w] = __fdiv_rn(t[w], b[w]);
        }
        lane_run<P, I + 1, next>(s);
    }
}

__device__ __forceinline__ void lane_wait(uint32_t depth)   // until at most depth - 2 groups of copies are on their way
{
    if (depth == 2) asm volatile("cp.async.wait_group 0;" ::: "memory");
    else if (depth == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 2;" ::: "memory");
}

/* Shared memory: per warp [depth stages of n_in tiles | n_out tiles]. */
template <class P> __device__ __forceinline__ void lanes_body(const LaneArgs &a)
{
    using L = LaneProgram<P>;
    const int lane = threadIdx.x & 31;
    const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    char *const own = g_form_smem + warp * (a.depth * L::n_in + L::n_out) * kLaneTileBytes;
    const uint32_t own_address = (uint32_t)__cvta_generic_to_shared(own);
    const uint32_t step = gridDim.x * warps;
    uint32_t now = blockIdx.x * warps + warp, ask = now, stage = 0;
    auto issue = [&](uint32_t to_stage) {
        if (ask < a.count) {
            const uint32_t tile = a.first + ask;
#pragma unroll
            for (int k = 0; k < L::n_in; k++) {
                constexpr uint32_t loads = L::loads;
                const int t = L::slot(loads, k), left = a.rows[t] - (int)(tile * 32u);
                const char *from = reinterpret_cast<const char *>(a.base[t]) + 4ull * tile * 32u * a.stride[t];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int m = (lane + 32 * i) >> 2, c = lane & 3;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                                 ::"r"(own_address + (to_stage * L::n_in + k) * kLaneTileBytes + 16u * lane_position(m, c)),
                                 "l"(from + (m < left ? 4ull * m * a.stride[t] + 16u * c : 0ull)), "r"(m < left ? 16 : 0) : "memory");   // (rows that are not there: zeros)
                }
            }
        }
        ask += step;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (uint32_t d = 0; d + 1 < a.depth; d++) issue(d);
    char *const result = own + a.depth * L::n_in * kLaneTileBytes;
    for (; now < a.count; now += step) {
        lane_wait(a.depth);
        __syncwarp();   // the stage is complete, and every lane is done with the one before it and with the result tiles
        issue(stage == 0 ? a.depth - 1u : stage - 1u);
        LaneState<P> s;
#pragma unroll
        for (int k = 0; k < L::n_in; k++)
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const float4 v = *reinterpret_cast<const float4 *>(own + (stage * L::n_in + k) * kLaneTileBytes + 16 * lane_position(lane, c));
                s.in[k][c][0] = v.x; s.in[k][c][1] = v.y; s.in[k][c][2] = v.z; s.in[k][c][3] = v.w;
            }
        lane_run<P, 0, 0>(s);
#pragma unroll
        for (int k = 0; k < L::n_out; k++)
#pragma unroll
            for (int c = 0; c < 4; c++)
                *reinterpret_cast<float4 *>(result + k * kLaneTileBytes + 16 * lane_position(lane, c)) = make_float4(s.out[k][c][0], s.out[k][c][1], s.out[k][c][2], s.out[k][c][3]);
        __syncwarp();
        const uint32_t tile = a.first + now;
#pragma unroll
        for (int k = 0; k < L::n_out; k++) {
            constexpr uint32_t stores = L::stores;
            const int t = L::slot(stores, k), left = a.rows[t] - (int)(tile * 32u);
            char *to = reinterpret_cast<char *>(a.base[t]) + 4ull * tile * 32u * a.stride[t];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int m = (lane + 32 * i) >> 2, c = lane & 3;
                const float4 v = *reinterpret_cast<const float4 *>(result + k * kLaneTileBytes + 16 * lane_position(m, c));
                if (m < left) *reinterpret_cast<float4 *>(to + 4ull * m * a.stride[t] + 16u * c) = v;
            }
        }
        stage = stage + 1u == a.depth ? 0u : stage + 1u;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

}  // namespace gint

#define GINT_DEFINE_LANE_KERNEL(name)                                                                                                          \
    extern "C" __global__ void __launch_bounds__(512) gint_form_lanes_##name(const __grid_constant__ gint::LaneArgs a) { gint::lanes_body<gint::LaneCode_##name>(a); }
