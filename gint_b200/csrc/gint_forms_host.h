/*
 * gint_forms_host.h -- host side of the form kernels: recognises the program shapes that have a kernel of their own and lays out
 * their launches. Included by gint_capi.cu only, after gint_wide_host.h.
 */
#pragma once

#include <utility>

#include "gint_form_types.h"
#include "gint_lane_programs.h"

namespace {

enum { FORM_NONE = 0, FORM_ROWS = 1, FORM_LANES = 2, FORM_HEADS = 3, FORM_FLAT = 4 };

struct Form {
    int kind = FORM_NONE;
    int tensor[gint::ROWS_N_SLOTS] = {-1, -1, -1, -1};   // tensor slot of every operand of the form; -1: none
    int store = 0;                                       // which of them is stored to
    uint64_t extent[gint::ROWS_N_SLOTS] = {};            // bytes from the base pointer that the operand's accesses reach
    int gather_digit[gint::ROWS_N_SLOTS] = {};           // digit that is the slot's innermost batch dimension; -1: it has one entry
    bool gathers[gint::ROWS_N_SLOTS] = {};               // ... whose stride is not 0: an index chooses among its rows
    uint32_t base_align = 3;                             // alignment of the base pointers (minus 1)
    gint::RowsArgs rows;                                 // all but pointers, range and shared memory
    /* lane programs: which one, its slots, the tiles of the block grid */
    int lane_program = 0;
    uint32_t lane_loads = 0, lane_stores = 0, lane_tiles = 0;
    uint64_t lane_reach[GINT_MAX_TENSORS] = {};
    gint::LaneArgs lanes;
    int head_kernel = 0;
    gint::HeadsArgs heads;
    /* flat: tensor[] holds x, y (-1: none), z */
    int flat_kernel = 0;
    uint32_t flat_n = 0, flat_step = 0, flat_grid = 0, flat_element_bytes = 0;
    gint::FlatArgs flat;
};
/* a launch on a form kernel */
struct FormLaunch {
    int kernel = 0;              // of GINT_FORM_KERNELS
    uint32_t grid = 0, threads = 0, smem = 0, warps_per_program = 0;
    gint::RowsArgs rows;
    gint::LaneArgs lanes;
    gint::HeadsArgs heads;
    gint::FlatArgs flat;
};

struct FormDim { uint32_t size, stride; bool batch0; };

/* The digits of a slot's place (decode_tiles in gint_interp.cuh), those of one value left out. Fails where the block grid cuts
 * dimension 1, or an element index could leave 31 bits. */
bool form_dims(const gint_tensor_info &ti, int t, int n, std::vector<FormDim> *dims, uint64_t *reach)
{
    dims->clear();
    if (ti.block_grid_dims[t][0] != 1) return false;
    const int64_t step2 = (int64_t)ti.block_grid_steps[t][1] * ti.block_shape_stride_2[t][1];
    if (step2 < 0 || step2 >= (1ll << 31)) return false;
    if (ti.block_grid_dims[t][1] != 1) dims->push_back(FormDim{(uint32_t)ti.block_grid_dims[t][1], (uint32_t)step2, false});
    for (int j = 0; j < 4; j++) {
        if (ti.batch_strides[t][j] < 0) return false;
        if (ti.batch_shape[t][j] != 1) dims->push_back(FormDim{(uint32_t)ti.batch_shape[t][j], (uint32_t)ti.batch_strides[t][j], j == 0});
    }
    uint64_t last = (uint64_t)n;
    for (const FormDim &d : *dims) {
        if (d.size < 1 || d.size >= (1u << 31)) return false;
        if (d.stride != 0 && (uint64_t)(d.size - 1) > (1ull << 31) / d.stride) return false;
        last += (uint64_t)(d.size - 1) * d.stride;
    }
    *reach = last;
    return last < (1ull << 31) - 8192;
}

void form_magic(uint32_t size, uint32_t *magic, uint32_t *shift)
{
    uint32_t l = 0;
    while ((1ull << l) < size) l++;
    *magic = (uint32_t)(((1ull << (31 + l)) + size - 1) / size);   // size in [2, 2^31): below 2^32; exact for numbers below 2^31
    *shift = l;
}

/* The slots' common digits. A slot whose strides are all 0 is the same for every logical program whatever its digits are. */
bool form_grid(const gint_tensor_info &ti, const int *tensor, int n_slots, const int *n, int elem_bytes, gint::FormGrid *grid, gint::FormSlot *slots, Form *f)
{
    std::vector<FormDim> common, dims;
    bool have = false;
    memset(grid, 0, sizeof(*grid));
    grid->gather_dim = -1;
    for (int s = 0; s < n_slots; s++) {
        slots[s] = gint::FormSlot{};
        if (tensor[s] < 0) continue;
        uint64_t reach = 0;
        if (ti.elm_size[tensor[s]] != elem_bytes || n[s] < 1 || !form_dims(ti, tensor[s], n[s], &dims, &reach)) return false;
        slots[s].n = n[s];
        f->extent[s] = reach * (uint64_t)elem_bytes;
        bool moves = false;
        for (const FormDim &d : dims) moves = moves || d.stride != 0;
        f->gather_digit[s] = -1;
        f->gathers[s] = ti.batch_strides[tensor[s]][0] != 0;
        for (size_t j = 0; j < dims.size(); j++) if (dims[j].batch0) f->gather_digit[s] = (int)j;
        slots[s].stationary = !moves;
        if (!moves) continue;
        if (have && dims.size() != common.size()) return false;
        for (size_t j = 0; have && j < dims.size(); j++) if (dims[j].size != common[j].size) return false;
        common = dims;
        have = true;
        for (size_t j = 0; j < dims.size(); j++) slots[s].stride[j] = dims[j].stride;
    }
    grid->n_dims = (uint32_t)common.size();
    for (size_t j = 0; j < common.size(); j++) {
        grid->size[j] = common[j].size;
        form_magic(common[j].size, &grid->magic[j], &grid->shift[j]);
    }
    return true;
}

/* what stands between the loops, as steps on the one value of the stack */
bool rows_steps(const std::vector<Insn> &p, size_t from, size_t to, gint::RowsArgs *a)
{
    a->n_steps = 0;
    for (size_t i = from; i < to; i++) {
        if (p[i].op == WOP_Remap) continue;   // (the form works in the natural layout)
        if (a->n_steps == gint::kRowsSteps) return false;
        uint32_t step = (uint32_t)p[i].op, operand = p[i].operand;
        if (p[i].op == OP_Dup && i + 2 < to && p[i + 1].op == OP_FPermW && p[i + 2].op == OP_FAdd) {
            step = gint::kRowsFold;
            operand = p[i + 1].operand;
            i += 2;
        } else if (p[i].op != OP_WarpAllReduceSum && p[i].op != OP_FAddImm && p[i].op != OP_FMulImm && p[i].op != OP_FMAImm && p[i].op != OP_FNeg &&
                   p[i].op != OP_FRSqrt && p[i].op != OP_FSqrt && p[i].op != OP_FRcp) return false;
        a->step[a->n_steps] = step;
        a->operand[a->n_steps++] = operand;
    }
    bool total = a->n_steps >= 3 && a->step[0] == OP_WarpAllReduceSum && a->step[1] == gint::kRowsFold && a->operand[1] == 0x01000302u &&
                 a->step[2] == gint::kRowsFold && a->operand[2] == 0x02030001u;
    for (uint32_t k = 3; k < a->n_steps; k++) total = total && a->step[k] != OP_WarpAllReduceSum && a->step[k] != gint::kRowsFold;
    const bool mean = total && a->n_steps == 6 && a->step[3] == OP_FMulImm && a->step[4] == OP_FAddImm && a->step[5] == OP_FRSqrt;
    a->steps = !total ? gint::STEPS_ANY : mean ? gint::STEPS_MEAN : a->n_steps == 3 ? gint::STEPS_TOTAL : gint::STEPS_TOTAL_THEN;
    return true;
}

/*
 * Row programs of f32 tiles: a running sum over the tiles of x (terms x, x * x, or fma(x, x)), steps on it, then either its store as
 * a tile or a second loop over the same tiles that stores
 *     s * x  [* w]  [silu]  [+ r]
 * Every operand's tiles start at element 0 of its row and are contiguous.
 */
bool match_rows(const std::vector<Insn> &p, const gint_tensor_info &ti, Form *f)
{
    gint::RowsArgs &a = f->rows;
    memset(&a, 0, sizeof(a));
    const int kLoad = GINT_W(LoadGlobal1DF32), kStore = GINT_W(StoreGlobal1DF32);
    for (int &t : f->tensor) t = -1;
    size_t i = 0;
    auto is = [&](int op) { return i < p.size() && p[i].op == op; };
    auto slot = [&](int s) {   // the operand of p[i]: element 0 of a slot
        const int t = (int)(p[i].operand & 15u);
        if ((p[i].operand >> 4) != 0 || t >= GINT_MAX_TENSORS || ti.block_shape_stride_1[t][1] != 1) return false;
        f->tensor[s] = t;
        i++;
        return true;
    };
    if (is(OP_LoadGlobal1DF32)) {   // two tiles are no loop: load, [square], load, [square], add
        const bool square = p.size() > 3 && p[1].op == OP_Dup;
        const size_t len = square ? 3 : 1;
        if (p.size() < 2 * len + 2 || !slot(gint::ROWS_X) || p[len].op != OP_LoadGlobal1DF32 || p[len].operand != p[0].operand + (128u << 4) || p[2 * len].op != OP_FAdd) return false;
        if (square && (p[2].op != OP_FMul || p[4].op != OP_Dup || p[5].op != OP_FMul)) return false;
        a.init = -0.0f;
        a.tiles = 2;
        a.reduce = square ? gint::ROWS_SUM_SQUARES : gint::ROWS_SUM;
        i = 2 * len + 1;
    } else {
        if (!is(OP_LoadImm)) return false;
        memcpy(&a.init, &p[i++].operand, 4);
        if (!is(WOP_LoopBegin) || p[i].operand == 0) return false;
        a.tiles = p[i++].operand;
        if (!is(kLoad) || !slot(gint::ROWS_X)) return false;
        if (is(WOP_AccAdd)) a.reduce = gint::ROWS_SUM;
        else if (is(WOP_AccFMASquare)) a.reduce = gint::ROWS_FMA_SQUARES;
        else if (is(WOP_Square)) {
            a.reduce = gint::ROWS_SUM_SQUARES;
            i++;
            if (!is(WOP_AccAdd)) return false;
        } else return false;
        i++;
        if (!is(WOP_LoopEnd)) return false;
        i++;
    }
    const size_t from = i;
    while (i < p.size() && p[i].op != WOP_LoopBegin && p[i].op != OP_StoreGlobal1DF32) i++;
    if (!rows_steps(p, from, i, &a)) return false;
    if (is(OP_StoreGlobal1DF32)) {
        const int t = (int)(p[i].operand & 15u);
        if (t >= GINT_MAX_TENSORS || (ti.block_shape_stride_1[t][1] != 1 && ti.block_shape_stride_1[t][0] != 1)) return false;
        f->tensor[gint::ROWS_Z] = t;
        a.store_at = (int)(p[i++].operand >> 4);
    } else {
        if (!is(WOP_LoopBegin) || p[i].operand != a.tiles) return false;
        i++;
        const int x = f->tensor[gint::ROWS_X];
        if (!is(kLoad) || !slot(gint::ROWS_X) || f->tensor[gint::ROWS_X] != x) return false;
        if (!is(WOP_MulKeep)) return false;
        i++;
        a.map = gint::ROWS_MAP;
        if (is(kLoad) && i + 1 < p.size() && p[i + 1].op == GINT_W(FMul)) {
            if (!slot(gint::ROWS_W)) return false;
            i++;
            a.map |= gint::ROWS_MAP_W;
        }
        if (is(WOP_Silu)) {
            memcpy(&a.silu, &p[i++].operand, 4);
            a.map |= gint::ROWS_MAP_SILU;
        }
        if (is(kLoad) && i + 1 < p.size() && p[i + 1].op == GINT_W(FAdd)) {
            if (!slot(gint::ROWS_R)) return false;
            i++;
            a.map |= gint::ROWS_MAP_R;
        }
        if (!is(kStore) || !slot(gint::ROWS_Z)) return false;
        if (!is(WOP_LoopEnd)) return false;
        i++;
        if (is(OP_Pop)) i++;
    }
    if (!is(OP_Halt)) return false;
    int n[gint::ROWS_N_SLOTS] = {};
    for (int s = 0; s < gint::ROWS_N_SLOTS; s++) {
        if (f->tensor[s] < 0) continue;
        n[s] = ti.block_shape_stride_1[f->tensor[s]][0];
        if (s != gint::ROWS_Z && f->tensor[s] == f->tensor[gint::ROWS_Z]) return false;
    }
    f->store = gint::ROWS_Z;
    if (!form_grid(ti, f->tensor, gint::ROWS_N_SLOTS, n, 4, &a.grid, a.slot, f)) return false;
    a.full_tiles = a.tiles;
    uint32_t stage = 0;
    for (int s = 0; s < gint::ROWS_N_SLOTS; s++) {
        if (f->tensor[s] < 0) continue;
        if (s == gint::ROWS_Z && !a.map) break;
        if ((uint64_t)n[s] > 128ull * a.tiles) a.slot[s].n = (int)(128u * a.tiles);   // the elements that the program has to do with: what is staged, and what the kernels' masks go by
        if ((uint32_t)n[s] / 128u < a.full_tiles) a.full_tiles = (uint32_t)n[s] / 128u;
        if (s == gint::ROWS_Z) break;
        uint32_t &area = a.slot[s].stationary ? a.stationary_bytes : stage;
        if (a.slot[s].n > 65536) return false;
        a.slot[s].area = area;
        area += (((uint32_t)a.slot[s].n * 4u + 15u) & ~15u) + 16u;   // a row may start anywhere in its first 16 bytes
    }
    a.fours = a.map != 0 && n[gint::ROWS_Z] % 4 == 0;
    for (int s = 0; s < gint::ROWS_N_SLOTS; s++) {
        if (f->tensor[s] < 0) continue;
        a.fours = a.fours && n[s] == n[gint::ROWS_Z];
        for (uint32_t stride : a.slot[s].stride) a.fours = a.fours && stride % 4 == 0;
    }
    a.stage_bytes = stage + 16u;                                  // ... and the stage's note of where its rows start
    f->kind = FORM_ROWS;
    return true;
}

/* of GINT_FORM_KERNELS: two per shape, the first of them with one warp per logical program */
int rows_kernel(const gint::RowsArgs &a)
{
    int k = 0;
#define GINT_X_SHAPE(name, r, m, s)                                                                                                              \
    if ((gint::Rows_##name::map < 0) || (a.reduce == (uint32_t)gint::Rows_##name::reduce && a.map == (uint32_t)gint::Rows_##name::map && a.steps == (uint32_t)gint::Rows_##name::steps)) return k; \
    k += 2;
    using namespace gint;
    GINT_ROWS_SHAPES(GINT_X_SHAPE)
#undef GINT_X_SHAPE
    return k - 2;
}

/*
 * Team size, teams per block and stages per team; every team has two to four stages (one computed, the others on their way), and there are no
 * more teams than rows. Measured (one B200, us per launch back to back, cold buffers, floor = bytes at 6557 GB/s; both sides of a line at the step that drew it, those of
 * SiLU with a residual of which L2 held a part):
 *
 * A pass that only scales is bound by memory, and memory serves it best with about 100 KB of rows per SM staged, two or three per team: more
 * rows at once are more pages read and written in turn. RMSNorm 16384 x 4096 86 with 98 KB, 91 with 197 KB (floor 82), 30 000 x 2048 78 and
 * 88 (75), 20 000 x 3072 78 and 85 (75), 13 000 x 6000 102 and 107 (95), 40 000 x 1536 78 and 93 (75), 60 000 x 1025 80 and 94 (75); one warp
 * per row of aligned rows 90 KB (100 000 x 768 101 with 74 KB, 110 with 98 KB, 100 000 x 700 94 with 90 KB, 102 with 112 KB).
 * Four warps per row from 1400 elements on (40 000 x 1535 one warp 91, four 80; 60 000 x 1025 80 and 104), four elements at a time from
 * 1000 on (60 000 x 1024 80 and 77; 80 000 x 900 94 and 103).
 *
 * SiLU is bound by issue: as many warps as have two stages, a multiple of four of them (one per scheduler and round: 65536 x 1024 118 with
 * 12, 129 with 13), one per row where that makes eight of them, or twelve if they go one element at a time (30 000 x 1536 88 with 8, four
 * per row 98; 38 000 x 1301 150 with 8, four per row 136; 12 000 x 4096 four per row 85, one 140).
 *
 * Sums: all the warps that have two stages. Rows of two or three tiles gain up to 32 warps (RMSNorm 600 000 x 129 335 with 16, 236 with 24,
 * 225) and up to four stages (300 000 x 256 104 with two, 98). At most two rows per SM: four warps per row (silu 100 x 1024 13, one warp 17).
 *
 * What is chosen measures now: RMSNorm 16384 x 4096 86, 30 000 x 2048 78, 20 000 x 3072 78, 13 000 x 6000 101, 40 000 x 1536 79, 40 000 x 1535 80, 60 000 x 1024
 * 80, 80 000 x 900 93, 100 000 x 768 100, 300 000 x 256 97, 600 000 x 129 215; silu + residual 65536 x 1024 139 (floor 123), 12 000 x 4096 98 (90), 30 000 x 1536
 * 92 (85), 38 000 x 1301 132, 150 000 x 300 117 (83), 100 x 1024 6.5.
 *
 * Left to the interpreter: SiLU with one team per SM (8000 x 8192 213 here, 187 there); rows of which two and the stationary ones
 * do not fit (RMSNorm of 20 000 values).
 */
struct RowsPlan { uint32_t team, teams, depth, grid, smem; };
bool plan_rows(const gint::RowsArgs &a, uint32_t count, int sms, int max_smem, RowsPlan *plan)
{
    const uint32_t exchange = 1024u, barriers = 32u;   // per team
    if ((uint64_t)a.stationary_bytes + 16u + 2ull * a.stage_bytes + exchange + barriers > (uint64_t)max_smem) return false;
    const uint32_t room = (uint32_t)max_smem - a.stationary_bytes - 16u, need = (count + (uint32_t)sms - 1) / (uint32_t)sms;
    const uint32_t one = room / (2u * a.stage_bytes + barriers);   // teams of one warp that have two stages
    const bool silu = (a.map & gint::ROWS_MAP_SILU) != 0, scales = a.map && !silu;
    const bool fours = a.fours && gint::kRowsShapes[rows_kernel(a) / 2].fours;
    uint32_t row_bytes = 0;   // of a stage
    for (int s = 0; s < gint::ROWS_Z; s++)
        if (!a.slot[s].stationary) row_bytes += 4u * (uint32_t)a.slot[s].n;
    bool four;
    if (a.tiles < 4) four = false;
    else if (need <= 2) four = true;
    else if (scales) four = a.slot[gint::ROWS_X].n >= (fours ? 1000 : 1400);
    else four = one < (silu && fours ? 8u : 12u);
    plan->team = four ? 4 : 1;
    const uint32_t extra = (four ? exchange : 0u) + barriers, best = four || !fours ? 100u * 1024u : 90u * 1024u;
    uint32_t t = need < (four ? 8u : 32u) ? need : four ? 8u : 32u;
    if (scales && t > 1 && t * 2u * row_bytes > best) t = best / (2u * row_bytes) ? best / (2u * row_bytes) : 1u;
    while (t > 1 && t * (2 * a.stage_bytes + extra) > room) t--;
    if (!four && a.map && t > 4) t &= ~3u;
    if (silu && t == 1 && need > 2u) return false;
    uint32_t d = (room - t * extra) / (t * a.stage_bytes);
    if (scales && a.tiles > 3 && d > best / (t * row_bytes + 1u)) d = best / (t * row_bytes + 1u);
    plan->teams = t;
    plan->depth = d > 4 ? 4 : d < 2 ? 2 : d;
    plan->smem = a.stationary_bytes + 16u + t * (plan->depth * a.stage_bytes + extra);
    const uint32_t blocks = (count + t - 1) / t;
    plan->grid = blocks < (uint32_t)sms ? blocks : (uint32_t)sms;
    return true;
}

/*
 * Lane programs (gint_lanes.cuh): exactly the instructions of a program that was compiled ahead of time, over rows of 16 floats whose accesses
 * are never masked along the row, and a block grid that steps by whole tiles of 32 rows.
 */
struct LaneCode { const int (*code)[2]; int n; };
#define GINT_X_LANE(name) {gint::LaneCode_##name::code, gint::LaneCode_##name::n},
const LaneCode kLanePrograms[] = {GINT_LANE_PROGRAMS(GINT_X_LANE)};
#undef GINT_X_LANE
constexpr int kLaneKernelFirst = 8;   // of GINT_FORM_KERNELS

bool match_lanes(const std::vector<Insn> &p, const gint_tensor_info &ti, int n_tensors, int pool_size, Form *f)
{
    int found = -1;
    for (size_t k = 0; k < sizeof(kLanePrograms) / sizeof(kLanePrograms[0]); k++) {
        const LaneCode &c = kLanePrograms[k];
        bool same = (size_t)c.n == p.size();
        for (size_t i = 0; same && i < p.size(); i++) same = p[i].op == c.code[i][0] && (!GINT_OP_USES_OPERAND(p[i].op) || p[i].operand == (uint32_t)c.code[i][1]);
        if (same) found = (int)k;
    }
    if (found < 0 || !rf_equivalent(p, pool_size)) return false;   // (the compiled program keeps its registers apart from the stack)
    f->lane_loads = f->lane_stores = f->lane_tiles = 0;
    for (const Insn &x : p)
        if (is_tensor_op(x.op)) (writes_tensor(x.op) ? f->lane_stores : f->lane_loads) |= 1u << (x.operand & 15u);
    if (f->lane_loads & f->lane_stores) return false;
    memset(&f->lanes, 0, sizeof(f->lanes));
    for (int t = 0; t < n_tensors; t++) {
        if (!(((f->lane_loads | f->lane_stores) >> t) & 1u)) continue;
        const int64_t rows = ti.block_shape_stride_1[t][0], stride = ti.block_shape_stride_1[t][1], tiles = ti.block_grid_dims[t][0];
        if (ti.elm_size[t] != 4 || ti.block_shape_stride_2[t][0] < 16 || ti.block_shape_stride_2[t][1] != 1 || rows < 1 || tiles < 1) return false;
        if (stride < 16 || stride % 4 != 0 || (tiles > 1 && ti.block_grid_steps[t][0] != 32) || ti.block_grid_dims[t][1] != 1) return false;
        for (int j = 0; j < 4; j++) if (ti.batch_shape[t][j] != 1) return false;
        if (f->lane_tiles && f->lane_tiles != (uint32_t)tiles) return false;
        if ((rows + 32) * stride >= (1ll << 31) || tiles * 32 >= (1ll << 31)) return false;
        f->lane_tiles = (uint32_t)tiles;
        f->lane_reach[t] = 4ull * (uint64_t)((rows - 1) * stride + 16);
        f->lanes.stride[t] = (uint32_t)stride;
        f->lanes.rows[t] = (int)rows;
    }
    f->lane_program = found;
    f->kind = FORM_LANES;
    return true;
}

/* Launches that L2 holds: 16 warps per SM with up to four stages. Larger ones: 12 with as many as make 84 KB of tiles, two at least -- as with rows
 * (plan_rows), more tiles at once are slower. Measured (one B200, us, back to back): product of 4 194 304 matrices 122 with 12 x 2 stages, 128 with 16 x 2,
 * 131 with 16 x 3 (floor 123); inverse 88 with 12 x 3, 94 with 12 x 4, 98 with 16 x 3, 100 with 16 x 4 (floor 82); of 300 000 the product 13.3
 * and 12.4. Fewer tiles than warps: fewer warps. */
bool plan_lanes(const Form &f, uint32_t count, int sms, int max_smem, FormLaunch *l)
{
    const uint32_t n_in = (uint32_t)__builtin_popcount(f.lane_loads), n_out = (uint32_t)__builtin_popcount(f.lane_stores);
    const bool large = (uint64_t)count * (n_in + n_out) * gint::kLaneTileBytes > (100ull << 20);
    uint32_t w = (count + (uint32_t)sms - 1) / (uint32_t)sms;
    if (w > (large ? 12u : 16u)) w = large ? 12u : 16u;
    const uint32_t tiles = (uint32_t)max_smem / w / gint::kLaneTileBytes;
    if (tiles < 2 * n_in + n_out) return false;
    uint32_t d = (tiles - n_out) / n_in;
    if (large && d > 84u * 1024u / (w * n_in * gint::kLaneTileBytes)) d = 84u * 1024u / (w * n_in * gint::kLaneTileBytes);
    l->lanes.depth = d > 4 ? 4 : d < 2 ? 2 : d;
    l->smem = w * (l->lanes.depth * n_in + n_out) * gint::kLaneTileBytes;
    l->threads = w * 32u;
    const uint32_t blocks = (count + w - 1) / w;
    l->grid = blocks < (uint32_t)sms ? blocks : (uint32_t)sms;
    l->warps_per_program = 1;
    return true;
}


/*
 * Normalisation of short bfloat16 rows, four per logical program (2DT tiles): a sum of squares by fma over two to four tiles of x, times a
 * factor plus an addend, 1 / sqrt, and y = (that * x) * w, w being one row for all.
 */
constexpr int kHeadsKernelFirst = 10;   // of GINT_FORM_KERNELS: rows of two tiles

bool match_heads(const std::vector<Insn> &p, const gint_tensor_info &ti, Form *f)
{
    gint::HeadsArgs &a = f->heads;
    memset(&a, 0, sizeof(a));
    for (int &t : f->tensor) t = -1;
    const int kLoad = GINT_W(LoadGlobal2DTBF16), kStore = GINT_W(StoreGlobal2DTBF16);
    size_t i = 0;
    auto take = [&](int op, uint32_t *operand) {
        if (i >= p.size() || p[i].op != op) return false;
        if (operand) *operand = p[i].operand;
        i++;
        return true;
    };
    uint32_t init, tiles, tiles2, x, x2, w, y, factor, addend;
    if (!take(OP_LoadImm, &init) || !take(WOP_LoopBegin, &tiles) || !take(kLoad, &x) || !take(WOP_AccFMASquare, nullptr) || !take(WOP_LoopEnd, nullptr)) return false;
    if (!take(OP_WarpAllReduceSum, nullptr)) return false;
    if (take(OP_FMAImm, &factor)) {
        a.fused = 1;
        a.factor = __half2float(__ushort_as_half((unsigned short)(factor & 0xFFFFu)));
        a.addend = __half2float(__ushort_as_half((unsigned short)(factor >> 16)));
    } else {
        if (!take(OP_FMulImm, &factor) || !take(OP_FAddImm, &addend)) return false;
        memcpy(&a.factor, &factor, 4);
        memcpy(&a.addend, &addend, 4);
    }
    if (!take(OP_FRSqrt, nullptr) || !take(WOP_LoopBegin, &tiles2) || !take(kLoad, &x2) || !take(WOP_MulKeep, nullptr) || !take(kLoad, &w) || !take(GINT_W(FMul), nullptr)) return false;
    if (!take(kStore, &y) || !take(WOP_LoopEnd, nullptr)) return false;
    take(OP_Pop, nullptr);
    if (!take(OP_Halt, nullptr)) return false;
    memcpy(&a.init, &init, 4);
    if (tiles < 2 || tiles > 4 || tiles2 != tiles || x2 != x || x >= GINT_MAX_TENSORS || w >= GINT_MAX_TENSORS || y >= GINT_MAX_TENSORS || y == x || y == w) return false;   // (offsets 0)
    const int tensor[3] = {(int)x, (int)w, (int)y}, n1 = ti.block_shape_stride_1[x][0];
    int n[3] = {n1, n1, n1};
    if (n1 <= 32 * ((int)tiles - 1)) return false;
    for (int t : tensor) {
        if (ti.block_shape_stride_1[t][0] != n1 || ti.block_shape_stride_1[t][1] != 1 || ti.block_shape_stride_2[t][1] < 0) return false;
        if (ti.block_shape_stride_2[t][0] != ti.block_shape_stride_2[x][0] || ti.block_grid_dims[t][1] != ti.block_grid_dims[x][1] || ti.block_grid_steps[t][1] != ti.block_grid_steps[x][1]) return false;
    }
    if (ti.block_shape_stride_2[w][1] != 0 || ti.block_shape_stride_2[x][0] < 1 || ti.block_grid_steps[x][1] < 0) return false;
    if ((int64_t)ti.block_grid_dims[x][1] * ti.block_grid_steps[x][1] >= (1ll << 31)) return false;
    if (!form_grid(ti, tensor, 3, n, 2, &a.grid, a.slot, f) || !a.slot[gint::HEADS_W].stationary) return false;
    for (int s = 0; s < 3; s++) {
        const int64_t stride2 = ti.block_shape_stride_2[tensor[s]][1];
        f->tensor[s] = tensor[s];
        /* four rows from the first one on, as far as there are rows */
        const int64_t begin = (int64_t)(ti.block_grid_dims[x][1] - 1) * ti.block_grid_steps[x][1], end = ti.block_shape_stride_2[x][0] - 1;
        f->extent[s] += (uint64_t)(2 * stride2 * (begin + 3 < end ? begin + 3 : end)) - (uint64_t)(2 * stride2 * begin);
        if (f->extent[s] / 2 >= (1ull << 31) - 8192) return false;
        a.row_stride[s] = (uint32_t)stride2;
    }
    if (ti.block_grid_dims[x][1] != 1) {
        if (a.grid.n_dims == 0 || a.grid.size[0] != (uint32_t)ti.block_grid_dims[x][1]) return false;   // (the slots that move share the digits)
        a.slot[gint::HEADS_ROW].stride[0] = (uint32_t)ti.block_grid_steps[x][1];
    }
    a.rows = ti.block_shape_stride_2[x][0];
    f->store = gint::HEADS_Y;
    /* four elements per lane and access: rows of 128, every offset of a row a multiple of 4 elements */
    bool fours = n1 == 128 && tiles == 4;
    for (int s = 0; s < 3; s++) {
        fours = fours && a.row_stride[s] % 4 == 0;
        for (uint32_t stride : a.slot[s].stride) fours = fours && stride % 4 == 0;
    }
    f->head_kernel = kHeadsKernelFirst + (fours ? 3 : (int)tiles - 2);
    f->kind = FORM_HEADS;
    return true;
}

/* The digits in the order of the strides of x, so that logical programs that follow one another lie next to one another. For launches of
 * the whole grid, which is the same set of logical programs in any order. */
void sort_digits(gint::HeadsArgs *a)
{
    gint::FormGrid &g = a->grid;
    for (uint32_t i = 1; i < g.n_dims; i++)
        for (uint32_t j = i; j > 0 && a->slot[gint::HEADS_X].stride[j] < a->slot[gint::HEADS_X].stride[j - 1]; j--) {
            std::swap(g.size[j], g.size[j - 1]);
            std::swap(g.magic[j], g.magic[j - 1]);
            std::swap(g.shift[j], g.shift[j - 1]);
            for (gint::FormSlot &s : a->slot) std::swap(s.stride[j], s.stride[j - 1]);
        }
}


/* [silu](x) [+ y | * y] as one flat loop (WideStream::flat_tiles) over slots of one length and type, from element 0 on. */
constexpr int kFlatKernelFirst = 14;   // of GINT_FORM_KERNELS: f32, f16, bf16

bool match_flat(const WideStream &ws, const gint_tensor_info &ti, Form *f)
{
    const std::vector<Insn> &p = ws.prog;
    const int loads[3] = {GINT_W(LoadGlobal1DF32), GINT_W(LoadGlobal1DF16), GINT_W(LoadGlobal1DBF16)};
    const int stores[3] = {GINT_W(StoreGlobal1DF32), GINT_W(StoreGlobal1DF16), GINT_W(StoreGlobal1DBF16)};
    memset(&f->flat, 0, sizeof(f->flat));
    for (int &t : f->tensor) t = -1;
    size_t i = 1;
    int type = 0;
    auto is = [&](int op) { return i < p.size() && p[i].op == op; };
    if (!ws.flat_tiles || p[0].op != WOP_LoopBegin) return false;
    while (type < 3 && !is(loads[type])) type++;
    if (type == 3) return false;
    f->tensor[0] = (int)p[i++].operand;
    if (is(WOP_Silu)) {
        memcpy(&f->flat.silu, &p[i++].operand, 4);
        f->flat.map |= gint::FLAT_SILU;
    }
    if (is(loads[type])) {
        f->tensor[1] = (int)p[i++].operand;
        if (!is(GINT_W(FAdd)) && !is(GINT_W(FMul))) return false;
        f->flat.map |= is(GINT_W(FAdd)) ? gint::FLAT_ADD : gint::FLAT_MUL;
        i++;
    }
    if (!f->flat.map || !is(stores[type])) return false;
    f->tensor[2] = (int)p[i++].operand;
    if (!is(WOP_LoopEnd) || i + 2 != p.size()) return false;
    f->flat_n = 0;
    for (int s = 0; s < 3; s++) {
        const int t = f->tensor[s];
        if (t < 0) continue;
        if (t >= GINT_MAX_TENSORS || ti.block_shape_stride_1[t][0] < 1 || ti.block_shape_stride_1[t][1] != 1 || ti.elm_size[t] != (type ? 2 : 4)) return false;   // (an offset makes it larger)
        if (f->flat_n && f->flat_n != (uint32_t)ti.block_shape_stride_1[t][0]) return false;
        f->flat_n = (uint32_t)ti.block_shape_stride_1[t][0];
    }
    if (f->tensor[2] == f->tensor[0] || f->tensor[2] == f->tensor[1]) return false;
    f->flat_step = ws.flat_tiles * 128u;
    f->flat_grid = ws.flat_grid;
    f->flat_kernel = kFlatKernelFirst + type;
    f->flat_element_bytes = type ? 2u : 4u;
    f->store = 2;
    f->kind = FORM_FLAT;
    return true;
}

}  // namespace
