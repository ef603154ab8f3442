/*
 * gint_rows.cuh -- row programs as one kernel: reduce a row, turn the sum into a factor, scale the row with it.
 *
 * Programs of this form (RMSNorm and its relatives, with what torch.compile fuses behind it; row sums) read a row twice and are a
 * few hundred bytecode instructions long. Interpreted, they are bound by instruction issue and instruction fetch: 127 warp
 * instructions per 128-value tile on the tile kernels (16384 rows of 4096: 114 us), and on the streaming kernels 33 instruction
 * cache misses and two memory round trips per row (10007 rows of 2029: 55 us; their bytes take 82 and 25 us). Here:
 *
 *   - One warp runs one logical program at a time, from shared memory: a ring of `depth` stages per warp holds the rows of the
 *     programs to come, brought in with bulk copies while the current one is computed, so that every row crosses from memory once
 *     and no load waits. Rows that all programs share (the weights) are staged once per block.
 *   - A row may start at any element: the copy takes the 16-byte groups that it touches, and the lanes read at 4-byte granularity.
 *   - Element e of a tile belongs to lane e % 32, width value e / 32, and the running sum takes the tiles in order: the layout and
 *     the order of the interpreter, so results are the same bits.
 *   - A team is one warp where enough of them have room for their stages, else four warps that take a width value each and share
 *     the row's stages (plan_rows in gint_forms_host.h has both sides).
 *
 * Measured (one B200, us per launch back to back, interpreter -> here): RMSNorm 16384 x 4096 113 -> 86 (6.3 TB/s), 10007 x 2029 53 -> 31,
 * 100 000 x 700 188 -> 97, 600 000 x 129 552 -> 215, 148 x 4096 15 -> 6.4; silu(rmsnorm) + residual of gathered rows 65536 x 1024
 * 171 -> 139 (5.8 TB/s), 12 000 x 4095 215 -> 99; sums of 65536 rows of 1024 52 -> 43.5, of 12 000 rows of 4095 49 -> 33, of 150 000 rows of 300
 * 71 -> 49. Long rows are bound by memory, rows of a few tiles by issue. What mattered, each at its step on the way there: a row's fixed cost (copies by
 * every thread with cp.async 42 -> 37 on the 2029s, steps in a loop over a switch 50 -> 38), the quotient of SiLU (gint_silu.cuh;
 * 155 -> 137), the number of rows on their way, and how much code lies between one row and the next: the usual shapes have kernels of their
 * own (GINT_ROWS_SHAPES), the one kernel for all of them was slower on short rows (600 000 x 129 285 with it, 236; sums of 300 93, 53).
 */
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "gint_form_types.h"
#include "gint_opcodes.h"
#include "gint_silu.cuh"

namespace gint {

extern __shared__ __align__(128) char g_form_smem[];

/* the entry of the row index that logical program r names (0 if the launch gathers nothing) */
__device__ __forceinline__ long long form_row(const FormGrid &g, uint32_t r)
{
    if (g.gather_dim < 0) return 0;
    if (g.simple) return __ldg(g.gather_index + r);
    for (int j = 0; j < g.gather_dim; j++) r = form_quotient(g, r, j);
    const uint32_t q = form_quotient(g, r, g.gather_dim);
    return __ldg(g.gather_index + (r - q * g.size[g.gather_dim]));
}
/* torch's rule for a negative index; one that is out of range all the same is clamped (decode_tiles in gint_interp.cuh) */
__device__ __forceinline__ long long form_clamp(const FormGrid &g, long long row)
{
    if (g.gather_dim < 0) return 0;
    if (row < 0) row += (long long)g.gather_rows;
    return row < 0 ? 0 : row >= (long long)g.gather_rows ? (long long)g.gather_rows - 1 : row;
}

/* Barriers of the bulk copies. A wait gives up after `limit` ns (RowsArgs::wait_ns; a copy takes a microsecond or two, more only where its page has to be
 * brought in first). */
__device__ __forceinline__ void bar_init(uint32_t bar) { asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, u64 limit)
{
    u64 begin = 0, now;
    for (;;) {
        for (int k = 0; k < 64; k++) {
            uint32_t done;
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                         : "=r"(done) : "r"(bar), "r"(parity) : "memory");
            if (done) return true;
        }
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        if (begin == 0) begin = now;
        else if (now - begin >= limit) return false;
    }
}
/* the 16-byte groups that n floats from p on touch */
__device__ __forceinline__ uint32_t row_bytes(u64 p, int n) { return ((uint32_t)(p & 15u) + 4u * (uint32_t)n + 15u) & ~15u; }
__device__ __forceinline__ void copy_row(uint32_t to, u64 p, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(to), "l"(p & ~15ull), "r"(bytes), "r"(bar) : "memory");
}

__device__ __forceinline__ float rows_pick(const float (&v)[4], uint32_t i) { return i == 0 ? v[0] : i == 1 ? v[1] : i == 2 ? v[2] : v[3]; }

/* A team of TEAM warps runs a logical program; its thread has 4 / TEAM of the four width values of its lane. */
template <int TEAM> struct Team {
    static constexpr int kValues = 4 / TEAM;
    int id, thread;        // team of the block, thread of the team
    float *exchange;       // two tiles of 128 values (teams of more than one warp)
    uint32_t turn;         // which of them the next exchange uses
    __device__ __forceinline__ void sync() const
    {
        if constexpr (TEAM == 1) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(id + 1), "n"(TEAM * 32) : "memory");
    }
    /* sync, and whether `ok` holds for all of the team (a vote alone orders no memory accesses) */
    __device__ __forceinline__ bool all(bool ok) const
    {
        if constexpr (TEAM == 1) {
            __syncwarp();
            return __all_sync(0xffffffffu, ok);
        }
        uint32_t r;
        asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %3, 0;\n\tbar.red.and.pred q, %1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                     : "=r"(r) : "r"(id + 1), "n"(TEAM * 32), "r"((uint32_t)ok) : "memory");
        return r != 0;
    }
    /* all four width values of the lane. (An exchange area is written again two exchanges later, when every warp has passed the
     * barrier behind its reads.) */
    __device__ __forceinline__ void exchange_all(const float (&s)[4 / TEAM], float (&v)[4])
    {
        float *area = exchange + turn + (thread & 31);
        turn ^= 128u;
#pragma unroll
        for (int w = 0; w < 4 / TEAM; w++) area[32 * ((thread >> 5) * (4 / TEAM) + w)] = s[w];
        sync();
#pragma unroll
        for (int w = 0; w < 4; w++) v[w] = area[32 * w];
    }
};

/* steps from `from` on that work on every value by itself, up to one that does not: what stands between the loops are instructions on
 * the one value of the stack, as the interpreter executes them. Returns the first step not done. */
template <int N> __device__ __forceinline__ uint32_t rows_each(const RowsArgs &a, uint32_t from, float (&s)[N])
{
    for (uint32_t k = from; k < a.n_steps; k++) {
        const uint32_t operand = a.operand[k];
        const float imm = __uint_as_float(operand);
        switch (a.step[k]) {
        case OP_FAddImm:
#pragma unroll
            for (int w = 0; w < N; w++) s[w] = __fadd_rn(s[w], imm);
            break;
        case OP_FMulImm:
#pragma unroll
            for (int w = 0; w < N; w++) s[w] = __fmul_rn(s[w], imm);
            break;
        case OP_FMAImm: {   // f16x2: multiplier, addend
            const float m = __half2float(__ushort_as_half((unsigned short)(operand & 0xFFFFu))), c = __half2float(__ushort_as_half((unsigned short)(operand >> 16)));
#pragma unroll
            for (int w = 0; w < N; w++) s[w] = __fmaf_rn(s[w], m, c);
            break;
        }
        case OP_FNeg:
#pragma unroll
            for (int w = 0; w < N; w++) s[w] = __uint_as_float(__float_as_uint(s[w]) ^ 0x80000000u);
            break;
        case OP_FRSqrt:
#pragma unroll
            for (int w = 0; w < N; w++) s[w] = rsqrtf(s[w]);
            break;
        case OP_FSqrt:
#pragma unroll
            for (int w = 0; w < N; w++) s[w] = __fsqrt_rn(s[w]);
            break;
        case OP_FRcp:
#pragma unroll
            for (int w = 0; w < N; w++) s[w] = __frcp_rn(s[w]);
            break;
        default: return k;
        }
    }
    return a.n_steps;
}
template <int TEAM, int STEPS> __device__ __forceinline__ void rows_steps(const RowsArgs &a, Team<TEAM> &team, float (&s)[4 / TEAM])
{
    constexpr int N = 4 / TEAM;
    if (STEPS != STEPS_ANY || a.steps != STEPS_ANY) {   // the usual beginning: the sum over lanes and width values, which is one value for all
        float v[4];
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1)
#pragma unroll
            for (int w = 0; w < N; w++) s[w] = __fadd_rn(s[w], __shfl_xor_sync(0xffffffffu, s[w], m));
        if constexpr (TEAM == 1) {   // (reducing the four together takes 8 shuffles instead of 20, but three more in a row: 100 000 x 512 97 -> 104 us)
#pragma unroll
            for (int w = 0; w < 4; w++) v[w] = s[w];
        } else {
            team.exchange_all(s, v);
        }
        /* every lane has the same four values, and the two foldings give every one of them the same total */
        const float t = __fadd_rn(__fadd_rn(v[0], v[2]), __fadd_rn(v[1], v[3]));
        float one[1] = {t};
        if (STEPS == STEPS_MEAN || (STEPS == STEPS_ANY && a.steps == STEPS_MEAN)) one[0] = rsqrtf(__fadd_rn(__fmul_rn(t, __uint_as_float(a.operand[3])), __uint_as_float(a.operand[4])));
        else if (STEPS == STEPS_ANY) rows_each<1>(a, 3u, one);
#pragma unroll
        for (int w = 0; w < N; w++) s[w] = one[0];
        return;
    }
    if constexpr (STEPS == STEPS_ANY) for (uint32_t k = rows_each<N>(a, 0u, s); k < a.n_steps; k = rows_each<N>(a, k + 1u, s)) {
        const uint32_t operand = a.operand[k];
        if (a.step[k] == kRowsFold) {   // Dup, FPermW, FAdd
            float v[4];
            if constexpr (TEAM == 1) {
#pragma unroll
                for (int w = 0; w < 4; w++) v[w] = s[w];
            } else {
                team.exchange_all(s, v);
            }
            const uint32_t sel = operand >> (8 * N * (team.thread >> 5));
#pragma unroll
            for (int w = 0; w < N; w++) s[w] = __fadd_rn(s[w], rows_pick(v, (sel >> (8 * w)) & 3u));
        } else {                        // WarpAllReduceSum
#pragma unroll
            for (int m = 16; m >= 1; m >>= 1)
#pragma unroll
                for (int w = 0; w < N; w++) s[w] = __fadd_rn(s[w], __shfl_xor_sync(0xffffffffu, s[w], m));
        }
    }
}

/* The thread's value i of tile k in a staged row is row[128 k + 32 i] (row: the thread's first element); `left`: elements of the
 * row from there on. MASKED: a group of tiles that reaches behind the row's whole tiles. */
template <bool MASKED> __device__ __forceinline__ float staged(const float *row, int e, int left) { return !MASKED || e < left ? row[e] : 0.0f; }

template <int REDUCE> __device__ __forceinline__ float rows_term(float x, float s)
{
    return REDUCE == ROWS_SUM ? __fadd_rn(x, s) : REDUCE == ROWS_SUM_SQUARES ? __fadd_rn(__fmul_rn(x, x), s) : __fmaf_rn(x, x, s);
}
template <int REDUCE, int N, int U, bool MASKED> __device__ __forceinline__ void reduce_tiles(const float *x, int left, int tiles, float (&s)[N])
{
    float v[U][N];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
        for (int i = 0; i < N; i++) v[u][i] = staged<MASKED>(x, u * 128 + i * 32, left);
#pragma unroll
    for (int u = 0; u < U; u++)
        if (!MASKED || u < tiles) {   // (a sum takes no terms of tiles that the program does not have)
#pragma unroll
            for (int i = 0; i < N; i++) s[i] = rows_term<REDUCE>(v[u][i], s[i]);
        }
}
template <int REDUCE, int N> __device__ __forceinline__ void rows_reduce(const RowsArgs &a, const float *x, int left, float (&s)[N])
{
    constexpr int U = N == 1 ? 8 : N == 2 ? 4 : 2;
    const int full = (int)a.full_tiles, tiles = (int)a.tiles;
    int k = 0;
    for (; k + U <= full; k += U) reduce_tiles<REDUCE, N, U, false>(x + k * 128, 0, 0, s);
    for (; k < tiles; k += U) reduce_tiles<REDUCE, N, U, true>(x + k * 128, left - k * 128, tiles - k, s);
}

/* U tiles of the second pass, their loads in front; `left`: elements from the thread's first one on in every row */
template <int MAP, int N, int U, bool MASKED>
__device__ __forceinline__ void map_tiles(const float *x, const float *wt, const float *r, float *z, const int (&left)[ROWS_N_SLOTS], float c, const float (&s)[N])
{
    float v[U][N], g[U][N], h[U][N];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int e = u * 128 + i * 32;
            v[u][i] = staged<MASKED>(x, e, left[ROWS_X]);
            g[u][i] = (MAP & ROWS_MAP_W) ? staged<MASKED>(wt, e, left[ROWS_W]) : 0.0f;
            h[u][i] = (MAP & ROWS_MAP_R) ? staged<MASKED>(r, e, left[ROWS_R]) : 0.0f;
        }
    float o[U * N];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
        for (int i = 0; i < N; i++) {
            o[u * N + i] = __fmul_rn(s[i], v[u][i]);
            if constexpr ((MAP & ROWS_MAP_W) != 0) o[u * N + i] = __fmul_rn(g[u][i], o[u * N + i]);
        }
    if constexpr ((MAP & ROWS_MAP_SILU) != 0) silu(o, c);
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
        for (int i = 0; i < N; i++) {
            if constexpr ((MAP & ROWS_MAP_R) != 0) o[u * N + i] = __fadd_rn(h[u][i], o[u * N + i]);
            if (!MASKED || u * 128 + i * 32 < left[ROWS_Z]) z[u * 128 + i * 32] = o[u * N + i];
        }
}
template <int MAP, int N>
__device__ __forceinline__ void rows_map(const RowsArgs &a, const float *x, const float *wt, const float *r, float *z, int at, const float (&s)[N])
{
    constexpr int U = N == 1 ? 4 : N == 2 ? 4 : 2;
    const int full = (int)a.full_tiles, tiles = (int)a.tiles;
    int k = 0, left[ROWS_N_SLOTS] = {};
    for (; k + U <= full; k += U) map_tiles<MAP, N, U, false>(x + k * 128, wt + k * 128, r + k * 128, z + k * 128, left, a.silu, s);
    for (; k < tiles; k += U) {
#pragma unroll
        for (int t = 0; t < ROWS_N_SLOTS; t++) left[t] = a.slot[t].n - at - k * 128;
        map_tiles<MAP, N, U, true>(x + k * 128, wt + k * 128, r + k * 128, z + k * 128, left, a.silu, s);
    }
}

/* The second pass four elements at a time, where s is one value and every row starts at a 16-byte boundary and has a multiple of four elements
 * (the same number in every operand): tiles go to the team's warps in turn, U of them together. */
template <int MAP, int TEAM>
__device__ __forceinline__ void rows_map_fours(const RowsArgs &a, const float *x, const float *wt, const float *r, float *z, int thread, float s)
{
    constexpr int U = 2, STEP = TEAM * 128;
    const int n = a.slot[ROWS_Z].n;
    for (int e = 4 * thread; e < n; e += U * STEP) {
        float o[4 * U];
        float4 v[U], g[U], h[U];
        const bool both = e + STEP < n;
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (u > 0 && !both) {
                v[u] = g[u] = h[u] = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
                continue;
            }
            v[u] = *reinterpret_cast<const float4 *>(x + e + u * STEP);
            if constexpr ((MAP & ROWS_MAP_W) != 0) g[u] = *reinterpret_cast<const float4 *>(wt + e + u * STEP);
            if constexpr ((MAP & ROWS_MAP_R) != 0) h[u] = *reinterpret_cast<const float4 *>(r + e + u * STEP);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            o[4 * u] = __fmul_rn(s, v[u].x); o[4 * u + 1] = __fmul_rn(s, v[u].y); o[4 * u + 2] = __fmul_rn(s, v[u].z); o[4 * u + 3] = __fmul_rn(s, v[u].w);
            if constexpr ((MAP & ROWS_MAP_W) != 0) {
                o[4 * u] = __fmul_rn(g[u].x, o[4 * u]); o[4 * u + 1] = __fmul_rn(g[u].y, o[4 * u + 1]);
                o[4 * u + 2] = __fmul_rn(g[u].z, o[4 * u + 2]); o[4 * u + 3] = __fmul_rn(g[u].w, o[4 * u + 3]);
            }
        }
        if constexpr ((MAP & ROWS_MAP_SILU) != 0) silu(o, a.silu);
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (u > 0 && !both) continue;
            if constexpr ((MAP & ROWS_MAP_R) != 0) {
                o[4 * u] = __fadd_rn(h[u].x, o[4 * u]); o[4 * u + 1] = __fadd_rn(h[u].y, o[4 * u + 1]);
                o[4 * u + 2] = __fadd_rn(h[u].z, o[4 * u + 2]); o[4 * u + 3] = __fadd_rn(h[u].w, o[4 * u + 3]);
            }
            *reinterpret_cast<float4 *>(z + e + u * STEP) = make_float4(o[4 * u], o[4 * u + 1], o[4 * u + 2], o[4 * u + 3]);
        }
    }
}

/* Shared memory: [stationary rows | per team: `depth` stages | teams of more than one warp: exchange areas | barriers: one of the
 * stationary rows, per team one per stage]. */
/* SHAPE: RowsAny, or a program's shape at compile time -- less code between one row and the next (plan in gint_forms_host.h) */
template <int TEAM, class SHAPE> __device__ __forceinline__ void rows_body(const RowsArgs &a)
{
    constexpr int N = 4 / TEAM;
    const uint32_t teams = blockDim.x / (TEAM * 32);
    Team<TEAM> team;
    team.id = (int)(threadIdx.x / (TEAM * 32));
    team.thread = (int)(threadIdx.x % (TEAM * 32));
    team.turn = 0;
    const uint32_t areas = a.stationary_bytes + teams * a.depth * a.stage_bytes;
    team.exchange = reinterpret_cast<float *>(g_form_smem + areas) + team.id * 256;
    const uint32_t smem = (uint32_t)__cvta_generic_to_shared(g_form_smem);
    const uint32_t own = a.stationary_bytes + (uint32_t)team.id * a.depth * a.stage_bytes;
    const uint32_t bars = smem + areas + (TEAM > 1 ? teams * 1024u : 0u), own_bars = bars + 8u + (uint32_t)team.id * a.depth * 8u;
    if (threadIdx.x == 0) {
        for (uint32_t k = 0; k <= teams * a.depth; k++) bar_init(bars + 8u * k);
        asm volatile("fence.mbarrier_init.release.cluster;\n\tfence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t bytes = 0;
#pragma unroll
        for (int t = 0; t < ROWS_Z; t++)
            if (a.slot[t].n && a.slot[t].stationary) bytes += row_bytes(a.slot[t].base, a.slot[t].n);
        bar_expect(bars, bytes);
#pragma unroll
        for (int t = 0; t < ROWS_Z; t++)
            if (a.slot[t].n && a.slot[t].stationary) copy_row(smem + a.slot[t].area, a.slot[t].base, row_bytes(a.slot[t].base, a.slot[t].n), bars);
    }
    const uint32_t step = gridDim.x * teams;
    uint32_t now = blockIdx.x + gridDim.x * (uint32_t)team.id;   // logical programs, relative to first: the one computed,
    uint32_t ask = now;                                          // ... and the next one to bring in
    /* Sums take the rows from the last to the first: whoever wrote the tensor just before did it the other way round, and its last rows are
     * still in L2 (sums behind silu(rmsnorm) + residual over 65536 rows of 1024: the pass 185 -> 179 us). */
    auto program = [&](uint32_t k) { return SHAPE::map == 0 ? a.first + (a.count - 1u - k) : a.first + k; };
    long long row = 0;
    if (team.thread == 0 && ask < a.count) row = form_row(a.grid, program(ask));
    auto issue = [&](uint32_t stage) {
        if (team.thread == 0 && ask < a.count) {
            const uint32_t to = smem + own + stage * a.stage_bytes, bar = own_bars + 8u * stage;
            uint32_t off[ROWS_N_SLOTS], bytes[ROWS_Z], sum = 0;
            form_offsets(a.grid, a.slot, program(ask), form_clamp(a.grid, row), off);
            /* the stage's note: where its rows start, and where the result goes */
            *reinterpret_cast<uint4 *>(g_form_smem + own + (stage + 1u) * a.stage_bytes - 16u) = make_uint4(off[ROWS_X], off[ROWS_W], off[ROWS_R], off[ROWS_Z]);
#pragma unroll
            for (int t = 0; t < ROWS_Z; t++) {
                bytes[t] = a.slot[t].n && !a.slot[t].stationary ? row_bytes(a.slot[t].base + 4ull * off[t], a.slot[t].n) : 0u;
                sum += bytes[t];
            }
            bar_expect(bar, sum);
#pragma unroll
            for (int t = 0; t < ROWS_Z; t++)
                if (bytes[t]) copy_row(to + a.slot[t].area, a.slot[t].base + 4ull * off[t], bytes[t], bar);
            row = ask + step < a.count ? form_row(a.grid, program(ask + step)) : 0;
        }
        ask += step;
    };
    for (uint32_t d = 0; d + 1 < a.depth; d++) issue(d);
    bool ok = bar_wait(bars, 0u, a.wait_ns) && a.wait_ns != 0;
    uint32_t stage = 0, parity = 0;
    const int at = (team.thread & 31) + 32 * N * (team.thread >> 5);   // the thread's first element of a tile: lane + 32 * width value
    for (; now < a.count; now += step) {
        ok = bar_wait(own_bars + 8u * stage, parity, a.wait_ns) && ok;
        if (!team.all(ok)) break;   // (also: every thread is done with the stage before this one)
        const uint4 note = *reinterpret_cast<const uint4 *>(g_form_smem + own + (stage + 1u) * a.stage_bytes - 16u);
        issue(stage == 0 ? a.depth - 1u : stage - 1u);
        const uint32_t off[ROWS_N_SLOTS] = {note.x, note.y, note.z, note.w};
        const float *in[ROWS_Z];
#pragma unroll
        for (int t = 0; t < ROWS_Z; t++) {
            const u64 p = a.slot[t].base + 4ull * off[t];   // (off is 0 for a stationary slot)
            in[t] = reinterpret_cast<const float *>(g_form_smem + (a.slot[t].stationary ? 0u : own + stage * a.stage_bytes) + a.slot[t].area + (uint32_t)(p & 15u)) + at;
        }
        float *z = reinterpret_cast<float *>(a.slot[ROWS_Z].base + 4ull * off[ROWS_Z]) + at;
        float s[N];
#pragma unroll
        for (int i = 0; i < N; i++) s[i] = a.init;
        const int left = a.slot[ROWS_X].n - at;
        if constexpr (SHAPE::reduce >= 0) rows_reduce<SHAPE::reduce, N>(a, in[ROWS_X], left, s);
        else if (a.reduce == ROWS_SUM) rows_reduce<ROWS_SUM, N>(a, in[ROWS_X], left, s);
        else if (a.reduce == ROWS_SUM_SQUARES) rows_reduce<ROWS_SUM_SQUARES, N>(a, in[ROWS_X], left, s);
        else rows_reduce<ROWS_FMA_SQUARES, N>(a, in[ROWS_X], left, s);
        rows_steps<TEAM, SHAPE::steps>(a, team, s);
        if constexpr (SHAPE::map > 0 && SHAPE::steps == STEPS_MEAN) {
            if (a.fours) rows_map_fours<SHAPE::map, TEAM>(a, in[ROWS_X] - at, in[ROWS_W] - at, in[ROWS_R] - at, z - at, team.thread, s[0]);
            else rows_map<SHAPE::map, N>(a, in[ROWS_X], in[ROWS_W], in[ROWS_R], z, at, s);
        } else if constexpr (SHAPE::map > 0) rows_map<SHAPE::map, N>(a, in[ROWS_X], in[ROWS_W], in[ROWS_R], z, at, s);
        else switch (SHAPE::map == 0 ? 0u : a.map) {
        case 0:
#pragma unroll
            for (int i = 0; i < N; i++)
                if (a.store_at + i * 32 < a.slot[ROWS_Z].n - at) z[a.store_at + i * 32] = s[i];
            break;
#define GINT_ROWS_MAP(m) case ROWS_MAP | (m): if constexpr (SHAPE::map < 0) rows_map<ROWS_MAP | (m), N>(a, in[ROWS_X], in[ROWS_W], in[ROWS_R], z, at, s); break;
        GINT_ROWS_MAP(0)
        GINT_ROWS_MAP(ROWS_MAP_W)
        GINT_ROWS_MAP(ROWS_MAP_R)
        GINT_ROWS_MAP(ROWS_MAP_W | ROWS_MAP_R)
        GINT_ROWS_MAP(ROWS_MAP_SILU)
        GINT_ROWS_MAP(ROWS_MAP_W | ROWS_MAP_SILU)
        GINT_ROWS_MAP(ROWS_MAP_SILU | ROWS_MAP_R)
        GINT_ROWS_MAP(ROWS_MAP_W | ROWS_MAP_SILU | ROWS_MAP_R)
#undef GINT_ROWS_MAP
        }
        if (++stage == a.depth) { stage = 0; parity ^= 1u; }
    }
    if (now < a.count && team.thread == 0) {   // gave up: the copies that are on their way get the usual time to end before the block does
        *a.gave_up = 1u;
        __threadfence_system();
        bar_wait(bars, 0u, kRowsWaitNs);
        for (; now < ask && now < a.count; now += step) {
            bar_wait(own_bars + 8u * stage, parity, kRowsWaitNs);
            if (++stage == a.depth) { stage = 0; parity ^= 1u; }
        }
    }
}

}  // namespace gint

/* One block per SM, of up to 32 teams of one warp or eight of four (plan_rows): at most 64 registers. Without the 1 the compiler takes the bound for two blocks
 * and 32 registers in some of them, and a small change elsewhere moves a kernel from one side to the other (RMSNorm 60 000 x 1024 140 us at
 * 32 registers, 78 at 48 to 52). */
#define GINT_DEFINE_ROWS_KERNELS(shape)                                                                                                          \
    extern "C" __global__ void __launch_bounds__(1024, 1) gint_form_rows1_##shape(const __grid_constant__ gint::RowsArgs a) { gint::rows_body<1, gint::Rows_##shape>(a); } \
    extern "C" __global__ void __launch_bounds__(1024, 1) gint_form_rows4_##shape(const __grid_constant__ gint::RowsArgs a) { gint::rows_body<4, gint::Rows_##shape>(a); }
