/*
 * gint_wide_host.h -- host side of the streaming kernels (gint_wide.cuh): finds the tile loops of a straight-line program again
 * and rewrites it as a stream with loops. Included by gint_capi.cu only (uses its Insn, kEffects and helpers).
 */
#pragma once

namespace {

struct WideStream {
    std::vector<Insn> prog;                        // opcodes of the streaming kernels' dispatch space; ends with Halt
    uint8_t alias_slots[GINT_MAX_TENSORS] = {};    // bit b of [a]: the order of accesses to slots a and b changed; they must not overlap
    int max_depth = 0;                             // pool slots needed
    int max_tiles = 0;                             // tiles of the longest loop
    uint32_t flat_tiles = 0;                       // tiles per logical program if the program is one flat loop, else 0
    uint32_t flat_grid = 0;                        // logical programs the flat form covers
    uint32_t access_bytes[GINT_MAX_TENSORS] = {};  // widest element with which the program accesses a slot
    bool slow_rows = false;                        // a row program that the streaming kernels run slower than the tile kernels
    uint8_t vector_alias[GINT_MAX_TENSORS] = {};   // ... of accesses in different loops, which the vector layout makes with other lanes
    bool vector = false;                           // the kernels in the vector layout may run it (base pointers aligned to 4 elements)
};

bool wide_is_2dt(int op) { return op >= OP_LoadGlobal2DTF32 && op <= OP_LoadGlobal2DTU8; }
int wide_element_bytes(int op)
{
    if (op == OP_LoadGlobal1DU8 || op == OP_LoadGlobal2DTU8 || op == OP_LoadGlobal2DWU8) return 1;
    const bool f32 = op == OP_LoadGlobal1DF32 || op == OP_StoreGlobal1DF32 || op == OP_LoadGlobal2DTF32 || op == OP_StoreGlobal2DTF32 ||
                     op == OP_LoadGlobal2DWF32 || op == OP_StoreGlobal2DWF32;
    return f32 ? 4 : 2;
}
/* instructions that a streaming kernel runs out of line, four values at a time (and WOP_Silu) */
bool wide_out_of_line(int op) { return op == OP_FDiv || op == OP_FRDiv || op == OP_FSqrt || op == OP_FRcp; }
bool wide_is_load(int op) { return GINT_WIDE_TILE_OP(op) && !writes_tensor(op); }

/* instruction `b` is instruction `a` one tile (times `tiles`) further on */
bool wide_repeats(const Insn &a, const Insn &b, int tiles)
{
    if (a.op != b.op) return false;
    if (!GINT_WIDE_TILE_OP(a.op)) return a.operand == b.operand || !GINT_OP_USES_OPERAND(a.op);
    const uint64_t step = wide_is_2dt(a.op) ? 32u : 128u;
    return b.operand == a.operand + (uint64_t)tiles * (step << 4);   // (no wrap: an offset has 28 bits, the one behind the last is 0)
}

/* One loop body, checked and rewritten: `body` holds format instructions, executed at stack depth d0. Fails if an instruction
 * has no wide form or touches what lies below the body's own stack other than by reading it or by adding to it. */
bool wide_body(const std::vector<Insn> &body, int d0, std::vector<Insn> *out, int *max_depth, int *accumulations)
{
    std::vector<Insn> b;
    for (size_t i = 0; i < body.size();) {       // sequences with a form of their own
        auto is = [&](size_t k, int op) { return i + k < body.size() && body[i + k].op == op; };
        if (is(0, OP_Dup) && i + 1 < body.size() && wide_is_load(body[i + 1].op) && (is(2, OP_FMul) || (is(2, OP_Swap) && is(3, OP_FMul)))) {
            b.push_back(body[i + 1]);
            b.push_back(Insn{WOP_MulKeep, 0u});
            i += is(2, OP_FMul) ? 3 : 4;
        } else if (is(0, OP_Dup) && is(1, OP_FNeg) && is(2, OP_FExp) && is(3, OP_FAddImm) && is(4, OP_FRDiv)) {
            b.push_back(Insn{WOP_Silu, body[i + 3].operand});
            i += 5;
        } else if (is(0, OP_Dup) && is(1, OP_FMul)) {
            b.push_back(Insn{WOP_Square, 0u});
            i += 2;
        } else b.push_back(body[i++]);
    }
    out->clear();
    *accumulations = 0;
    int d = d0, acc_reads = 0;
    auto reads_below = [&](int pos) { if (pos == d0 - 1) acc_reads = 1; return pos >= 0; };
    for (size_t i = 0; i < b.size(); i++) {
        const Insn &in = b[i];
        if (in.op == WOP_MulKeep) {                  // reads d-2, d-1; writes d-1
            if (d - 1 < d0 || !reads_below(d - 2)) return false;
            out->push_back(in);
        } else if (in.op == WOP_Silu || in.op == WOP_Square) {
            if (d - 1 < d0) return false;
            out->push_back(in);
        } else if (!GINT_WIDE_OP(in.op)) {
            return false;
        } else if (in.op == OP_Dup && i + 1 < b.size() && b[i + 1].op == OP_FMA && d - 2 == d0 - 1 && d0 >= 1) {   // acc, x: acc + x * x
            out->push_back(Insn{WOP_AccFMASquare, 0u});
            ++*accumulations;
            i++;
            d -= 1;
            continue;
        } else if (in.op == OP_FAdd && d - 2 == d0 - 1 && d0 >= 1) {
            out->push_back(Insn{WOP_AccAdd, 0u});
            ++*accumulations;
            d -= 1;
            continue;
        } else if (in.op == OP_FMA && d - 3 == d0 - 1 && d0 >= 1) {
            out->push_back(Insn{WOP_AccFMA, 0u});
            ++*accumulations;
            d -= 2;
            continue;
        } else {
            const int md = kEffects[in.op].min_depth, net = kEffects[in.op].net;
            if (in.op == OP_Dup) { if (!reads_below(d - 1)) return false; }
            else if (in.op == OP_Dup2) { if (!reads_below(d - 1) || !reads_below(d - 2)) return false; }
            else if (d - md < d0) return false;      // everything else consumes or rewrites what it reads
            out->push_back(Insn{GINT_WIDE_FIRST + in.op, in.operand});
            d += net;
        }
        if (d > *max_depth) *max_depth = d;
        if (d < d0) return false;
    }
    if (d != d0) return false;
    if (*accumulations && acc_reads) return false;   // the running value itself is also read
    if (*accumulations > 1) return false;            // U terms of one kind, then U of the other: not the program's order
    return true;
}

bool wide_strides_disjoint(const gint_tensor_info &ti, int t, bool two_d)
{
    const int64_t n1 = ti.block_shape_stride_1[t][0], s1 = ti.block_shape_stride_1[t][1];
    const int64_t n2 = ti.block_shape_stride_2[t][0], s2 = ti.block_shape_stride_2[t][1];
    if (s1 <= 0 && n1 > 1) return false;
    if (!two_d || n2 <= 1) return true;
    return s2 > 0 && (s2 >= s1 * n1 || s1 >= s2 * n2);
}

/* Accesses whose order the loop changes: tiles of one iteration group are all loaded before the first of them is stored, and
 * stores to two slots no longer alternate. Slots that a loop stores to must therefore not overlap any other slot it uses
 * (recorded, checked against the launch's address ranges); a slot that is stored to and accessed a second time must be accessed
 * at the same place with elements of the same width, so that every tile stays with itself (tile k in f16 covers the second half of
 * tile k / 2 in f32). */
bool wide_hazards(const std::vector<Insn> &body, const gint_tensor_info &ti, uint8_t *alias_slots)
{
    for (const Insn &s : body) {
        if (!writes_tensor(s.op)) continue;
        const int t = (int)(s.operand & 15u);
        if (!wide_strides_disjoint(ti, t, wide_is_2dt(s.op))) return false;
        for (const Insn &x : body) {
            if (!GINT_WIDE_TILE_OP(x.op) || &x == &s) continue;
            const int u = (int)(x.operand & 15u);
            if (u != t) alias_slots[u] |= (uint8_t)(1u << t);
            else if (x.operand != s.operand || wide_element_bytes(x.op) != wide_element_bytes(s.op) || wide_is_2dt(x.op) || wide_is_2dt(s.op)) return false;
        }
    }
    return true;
}

/*
 * May the kernels in the vector layout run the stream? Every group of four elements that a lane then accesses must be aligned
 * given an aligned base pointer: stride 1 along dimension 1, every offset that a logical program can have a multiple of 4
 * elements. And nothing may tell the layouts apart: decided by vec_transform on the stream with each loop body written once
 * (what holds after one pass of a body holds after any number). Where it asks for a rearrangement outside of loops the stream
 * gets a Remap. 2DT tiles are only taken in fours (a loop of 4 n tiles), and the one thing that may look across their lanes is a
 * sum over the warp: a lane then adds the terms of other elements than in the natural layout, and the same elements are summed. The
 * order of the additions is another one, so it is done for elements of 2 bytes alone; sums of f32 and u8 elements keep theirs.
 */
bool wide_vector(WideStream *ws, const gint_tensor_info &ti, int n_tensors)
{
    /* What a loop stores a later one may access with another lane than in the natural layout: two slots that meet in memory, or one
     * slot at offsets that are not whole groups of 128 elements apart. Within a loop an accessed tile stays with itself. */
    struct Access { int loop; bool store; uint32_t operand; };
    std::vector<Access> accesses;
    int loop = 0;
    for (const Insn &x : ws->prog) {
        if (x.op == WOP_LoopBegin) loop++;
        const int op = x.op - GINT_WIDE_FIRST;
        if (op >= 0 && GINT_WIDE_TILE_OP(op)) accesses.push_back(Access{loop, writes_tensor(op), x.operand});
    }
    for (const Access &s : accesses)
        for (const Access &x : accesses) {
            if (!s.store || x.loop == s.loop) continue;
            const uint32_t t = s.operand & 15u, u = x.operand & 15u;
            if (u != t) ws->vector_alias[u] |= (uint8_t)(1u << t);
            else if (((x.operand >> 4) - (s.operand >> 4)) % 128u != 0) return false;
        }
    std::vector<Insn> rep, marked;
    std::vector<size_t> origin;
    bool any_2dt = false, any_1d = false, accumulates = false, in_fours = true, two_bytes = true;
    auto emit = [&](int op, uint32_t operand, size_t from) { rep.push_back(Insn{op, operand}); origin.push_back(from); };
    for (size_t i = 0; i < ws->prog.size(); i++) {
        const Insn &x = ws->prog[i];
        if (x.op >= GINT_WIDE_FIRST) {
            const int op = x.op - GINT_WIDE_FIRST, t = (int)(x.operand & 15u);
            if (!GINT_WIDE_TILE_OP(op)) { emit(op, x.operand, i); continue; }
            const bool two = wide_is_2dt(op);
            (two ? any_2dt : any_1d) = true;
            if (wide_element_bytes(op) != 2 && !writes_tensor(op)) two_bytes = false;
            bool ok = t < n_tensors && ti.block_shape_stride_1[t][1] == 1 && ti.elm_size[t] == wide_element_bytes(op) && ((x.operand >> 4) & 3u) == 0;
            if (ok && ti.block_grid_dims[t][0] != 1 && ti.block_grid_steps[t][0] % 4 != 0) ok = false;
            if (ok && two && ti.block_shape_stride_2[t][1] % 4 != 0) ok = false;
            if (ok && ti.block_grid_dims[t][1] != 1 && ((int64_t)ti.block_grid_steps[t][1] * ti.block_shape_stride_2[t][1]) % 4 != 0) ok = false;
            for (int j = 0; j < 4; j++)
                if (ti.batch_shape[t][j] != 1 && ti.batch_strides[t][j] % 4 != 0) ok = false;
            if (!ok) return false;
            emit(writes_tensor(op) ? OP_StoreGlobal1DF32Fast : OP_LoadGlobal1DF32Fast, 0u, i);
        } else switch (x.op) {
        case WOP_LoopBegin: if (x.operand % 4u != 0) in_fours = false; break;
        case WOP_LoopEnd: break;
        /* (the addition that follows a sum stands for "after this loop's tiles": equal sums of two loops are two values) */
        case WOP_AccAdd: accumulates = true; emit(OP_FAdd, 0u, i); emit(OP_FAddImm, (uint32_t)i, i); break;
        case WOP_AccFMA: accumulates = true; emit(OP_FMA, 0u, i); emit(OP_FAddImm, (uint32_t)i, i); break;
        case WOP_AccFMASquare: accumulates = true; emit(OP_Dup, 0u, i); emit(OP_FMA, 0u, i); emit(OP_FAddImm, (uint32_t)i, i); break;
        case WOP_Square: emit(OP_Dup, 0u, i); emit(OP_FMul, 0u, i); break;
        case WOP_MulKeep: emit(OP_Swap, 0u, i); emit(OP_DupX1, 0u, i); emit(OP_FMul, 0u, i); break;   // [s, x] -> [x, s] -> [s, x, s] -> [s, s x]
        case WOP_Silu: emit(OP_Dup, 0u, i); emit(OP_FNeg, 0u, i); emit(OP_FExp, 0u, i); emit(OP_FAddImm, x.operand, i); emit(OP_FRDiv, 0u, i); break;
        default: emit(x.op, x.operand, i);
        }
    }
    if (any_1d == any_2dt || (any_2dt && accumulates && !(in_fours && two_bytes))) return false;
    int n_vector = 0, n_remaps = 0;
    if (!vec_transform(rep, &marked, &n_vector, &n_remaps, any_2dt)) return false;
    std::vector<size_t> remap_before;
    size_t k = 0;
    for (const Insn &m : marked) {
        if (m.op != OP_RemapVN) { k++; continue; }
        const size_t at = origin[k];
        if (ws->prog[at].op >= GINT_N_OPCODES) return false;                     // inside a loop
        if (any_2dt && ws->prog[at].op != OP_WarpAllReduceSum) return false;
        if (!any_2dt) remap_before.push_back(at);
    }
    for (size_t j = remap_before.size(); j-- > 0;) ws->prog.insert(ws->prog.begin() + (long)remap_before[j], Insn{WOP_Remap, 0u});
    return true;
}

/*
 * The program as a stream with loops, or false. At every instruction the shortest body that repeats at least twice, each time
 * one tile further on, becomes a loop. A sum whose first term is computed before the loop (x0, then + x1, + x2, ...) starts from
 * -0 instead, which adds nothing to any value, and the loop takes the first tile as well. What stands between loops runs on one
 * tile. A program qualifies if at least three quarters of its tile accesses are inside loops, it uses no virtual registers,
 * moves no tensor, and no element index of it leaves 31 bits.
 */
bool wide_transform(const std::vector<Insn> &in, const gint_tensor_info &ti, int n_tensors, WideStream *out)
{
    std::vector<Insn> prog = in;
    for (size_t i = 1; i < prog.size(); i++)
        if (wide_is_load(prog[i].op) && prog[i - 1].op == prog[i].op && prog[i - 1].operand == prog[i].operand) prog[i] = Insn{OP_Dup, 0u};
    const size_t n = prog.size() - 1;                 // without the Halt
    if (n == 0) return false;
    int n_mem = 0;
    uint32_t used = 0;
    for (size_t i = 0; i < n; i++) {
        if (!GINT_WIDE_NARROW_OP(prog[i].op)) return false;
        if (!is_tensor_op(prog[i].op)) continue;
        n_mem++;
        const int t = (int)(prog[i].operand & 15u), bytes = wide_element_bytes(prog[i].op);
        used |= 1u << t;
        if ((uint32_t)bytes > out->access_bytes[t]) out->access_bytes[t] = (uint32_t)bytes;
    }
    for (int t = 0; t < n_tensors; t++)
        if (((used >> t) & 1u) && (tensor_extent_bytes(ti, t) == 0 || tensor_extent_bytes(ti, t) / 4 >= (1ull << 31) - 8192)) return false;
    std::vector<Insn> &p = out->prog;
    p.clear();
    int depth = 0, peak = 0;
    size_t narrow_from = 0;                           // first instruction of p after the last loop
    for (size_t i = 0; i < n;) {
        size_t len = 0;
        int count = 1;
        for (size_t L = 2; L <= 48 && i + 2 * L <= n; L++) {
            int c = 1;
            for (;; c++) {
                bool same = i + (size_t)(c + 1) * L <= n;
                for (size_t j = 0; same && j < L; j++) same = wide_repeats(prog[i + j], prog[i + (size_t)c * L + j], c);
                if (!same) break;
            }
            if (c < 2) continue;
            bool tile = false;
            for (size_t j = 0; j < L; j++) tile = tile || GINT_WIDE_TILE_OP(prog[i + j].op);
            int net = 0;
            for (size_t j = 0; j < L; j++) net += kEffects[prog[i + j].op].net;
            if (tile && net == 0) { len = L; count = c; break; }
        }
        std::vector<Insn> body, wide;
        int body_depth = depth;
        int accumulations = 0;
        if (len) {
            body.assign(prog.begin() + (long)i, prog.begin() + (long)(i + len));
            if (!wide_body(body, depth, &wide, &body_depth, &accumulations) || !wide_hazards(body, ti, out->alias_slots)) len = 0;
        }
        if (!len) {
            const int post = depth + kEffects[prog[i].op].net;
            if (post > peak) peak = post;
            p.push_back(prog[i]);
            depth = post;
            i++;
            continue;
        }
        i += len * (size_t)count;
        /* (the body's one sum is its last instruction: what stands before it in the first tile's instructions touches nothing below) */
        if (accumulations == 1 && wide.back().op == WOP_AccAdd && p.size() - narrow_from >= len - 1) {
            const size_t first = p.size() - (len - 1);
            std::vector<Insn> from_first = body, from_first_wide;
            bool same = true;
            for (size_t j = 0; same && j + 1 < len; j++) same = wide_repeats(p[first + j], body[j], 1);
            for (size_t j = 0; same && j + 1 < len; j++) from_first[j].operand = p[first + j].operand;
            if (same && wide_body(from_first, depth, &from_first_wide, &body_depth, &accumulations)) {
                body = from_first;
                wide = from_first_wide;
                p.resize(first);
                p.push_back(Insn{OP_LoadImm, 0x80000000u});
                count++;
            }
        }
        p.push_back(Insn{WOP_LoopBegin, (uint32_t)count});
        p.insert(p.end(), wide.begin(), wide.end());
        p.push_back(Insn{WOP_LoopEnd, 0u});
        narrow_from = p.size();
        if (body_depth > peak) peak = body_depth;
        if (count > out->max_tiles) out->max_tiles = count;
    }
    /* a program without a loop that could be the body of one: a single tile per logical program */
    if (out->max_tiles == 0) {
        std::vector<Insn> body(prog.begin(), prog.begin() + (long)n), wide;
        int body_depth = 0;
        int accumulations = 0;
        if (!wide_body(body, 0, &wide, &body_depth, &accumulations) || !wide_hazards(body, ti, out->alias_slots)) return false;
        p.clear();
        p.push_back(Insn{WOP_LoopBegin, 1u});
        p.insert(p.end(), wide.begin(), wide.end());
        p.push_back(Insn{WOP_LoopEnd, 0u});
        peak = body_depth;
        out->max_tiles = 1;
    }
    int n_outside = 0;
    for (const Insn &x : p) n_outside += x.op < GINT_N_OPCODES && is_tensor_op(x.op);
    if (4 * n_outside > n_mem) return false;
    p.push_back(Insn{OP_Halt, 0u});
    out->max_depth = peak;
    /* flat: one loop over 1-D tiles and nothing else, logical program b starting where b - 1 ends */
    bool flat = p[0].op == WOP_LoopBegin && p[p.size() - 2].op == WOP_LoopEnd;
    for (size_t i = 1; i + 2 < p.size(); i++)
        flat = flat && p[i].op >= WOP_LoopBegin && p[i].op != WOP_LoopBegin && p[i].op != WOP_LoopEnd && !wide_is_2dt(p[i].op - GINT_WIDE_FIRST);
    uint32_t grid = 0;
    int64_t last_offset = 0;   // of the program as written; a flat loop adds up to the whole grid's elements to it
    for (size_t i = 0; i < n; i++)
        if (is_tensor_op(prog[i].op) && (int64_t)(prog[i].operand >> 4) > last_offset) last_offset = (int64_t)(prog[i].operand >> 4);
    for (int t = 0; flat && t < n_tensors; t++) {
        if (!((used >> t) & 1u)) continue;
        const int64_t gd1 = (uint32_t)ti.block_grid_dims[t][0];
        flat = (uint32_t)ti.block_grid_dims[t][1] == 1u && ti.block_grid_steps[t][0] == out->max_tiles * 128 && gd1 >= 1 &&
               gd1 * ti.block_grid_steps[t][0] + last_offset < (1ll << 31) - 8192 && (grid == 0 || grid == (uint32_t)gd1);
        for (int j = 0; j < 4; j++) flat = flat && ti.batch_shape[t][j] == 1;
        grid = (uint32_t)gd1;
    }
    if (flat && grid) {
        out->flat_tiles = (uint32_t)out->max_tiles;
        out->flat_grid = grid;
        p[0].operand = 0u;
    } else if (out->max_tiles == 1) return false;
    /* Row programs with out-of-line math in a loop (division, square root, SiLU) stay on the tile kernels: two rows per warp and 28
     * warps per SM hide those chains better than one row and 16 (silu(rmsnorm) + residual over 65536 rows of 1024, with its row
     * sums: 250 us there, 340 us here). */
    if (!out->flat_tiles)
        for (const Insn &x : p) {
            if (x.op == WOP_Silu || wide_out_of_line(x.op - GINT_WIDE_FIRST)) out->slow_rows = true;
        }
    out->vector = !out->slow_rows && n_outside == 0 && wide_vector(out, ti, n_tensors);   // (the streaming kernels do not run slow rows, and forms ask for no layout)
    return true;
}

/* Loops whose body is one of GINT_WIDE_LOOP_LIST become one instruction, its operands in the entries behind it. */
struct LoopDef { int num, depth, len; int ops[8]; };
enum { LAY_1D, LAY_2DT };   // (columns of the list that only the kernels use)
enum { DT_F32, DT_F16, DT_BF16 };
const LoopDef kLoops[] = {
#define GINT_X_LOOPDEF(name, num, expr, lay, dt, d0, len, ...) {num, d0, len, {__VA_ARGS__}},
    GINT_WIDE_LOOP_LIST(GINT_X_LOOPDEF)
#undef GINT_X_LOOPDEF
};

int wide_net_effect(int op)
{
    if (op >= GINT_WIDE_FIRST) return kEffects[op - GINT_WIDE_FIRST].net;
    if (op < GINT_N_OPCODES) return kEffects[op].net;
    return op == WOP_AccAdd || op == WOP_AccFMASquare ? -1 : op == WOP_AccFMA ? -2 : 0;
}

void wide_fuse_loops(std::vector<Insn> *prog)
{
    const std::vector<Insn> p = *prog;
    prog->clear();
    int depth = 0;
    for (size_t i = 0; i < p.size();) {
        const size_t begin = i;
        const LoopDef *hit = nullptr;
        if (p[begin].op == WOP_LoopBegin)
            for (const LoopDef &d : kLoops) {
                bool same = d.depth == depth && begin + (size_t)d.len + 1 < p.size() && p[begin + (size_t)d.len + 1].op == WOP_LoopEnd;
                for (int j = 0; same && j < d.len; j++) same = p[begin + 1 + (size_t)j].op == d.ops[j];
                if (same) { hit = &d; break; }
            }
        if (!hit) {
            depth += wide_net_effect(p[i].op);
            prog->push_back(p[i++]);
            continue;
        }
        prog->push_back(Insn{hit->num, p[begin].operand});
        for (int j = 0; j < hit->len; j++) {
            const int op = hit->ops[j];
            if (op == WOP_Silu || (op >= GINT_WIDE_FIRST && GINT_WIDE_TILE_OP(op - GINT_WIDE_FIRST))) prog->push_back(Insn{OP_CARRIER, p[begin + 1 + (size_t)j].operand});
        }
        i = begin + (size_t)hit->len + 2;
    }
}

}  // namespace
