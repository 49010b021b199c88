// stroke_verbs.cuh — how the verb-parallel strokes (stroke_verbs.cu, stroke_steps.cu) describe a
// verb: its flags, its curve units and the packed form of a general join.
#pragma once

#include "points.cuh"
#include "stroke_parts.cuh"
#include "stroke_verbs.h"

namespace lg {
namespace {

constexpr int KIND_NONE = 7;           // an unused slot
constexpr uint32_t KIND_MASK = 7;
constexpr uint32_t KIND_MNEC = 0x80;   // End/Close: a point merged into the sub-path's first
constexpr uint32_t KIND_GAP = 0x40;    // line verbs were dropped right before this verb
// Flags of a verb.
constexpr uint32_t VF_IRR = 1;         // irregular
constexpr uint32_t VF_FLAT1 = 2;       // its first kept point is a flattening step
constexpr uint32_t VF_FLATL = 4;       // the kept point before its last one is one
constexpr uint32_t VF_NK_SHIFT = 3;    // kept points, at most 3 (two bits)
constexpr uint32_t VF_TURN = 32;       // a quadratic split at a sharp turn
constexpr uint32_t VF_TOFIRST = 64;    // its first join's edge ids coincide (EF_SELF_EQ)
constexpr uint32_t VF_CUT = 128;       // cut in two runs at an interior general join
constexpr uint32_t VF_MERGED = 256;    // its end point merged: its last kept point is in `fin`
constexpr uint32_t VF_ENDFLAT = 512;   // and that one is a flattening step
constexpr uint32_t VF_TWO = VF_TURN | VF_CUT;
constexpr uint32_t VF_SECOND1 = 1024;  // of two units, the second is one step
// A curve of more steps than this leaves its path to the walk, which takes 32 steps at a time.
constexpr uint32_t MAX_SERIAL_STEPS = 1u << 15;

__device__ __forceinline__ bool is_segment(int k) {
    return k == LYON_VERB_LINE_TO || k == LYON_VERB_QUADRATIC_TO || k == LYON_VERB_CUBIC_TO;
}
__device__ __forceinline__ bool is_end(int k) {
    return k == LYON_VERB_END || k == LYON_VERB_CLOSE;
}
__device__ __forceinline__ uint32_t flags_nk(uint32_t f) { return (f >> VF_NK_SHIFT) & 3u; }

// ---- packed joins ---------------------------------------------------------------------------
// A general join: vertices (21 bits), relative ids the next edge starts from (2 + 2), triangles
// less vertices + 4 (3 bits: interior triangles less base vertices), whether the edge into it has
// equal ids. Joins with more vertices or invalid ids are not packed (their path is walked).
__device__ __forceinline__ bool pack_join(const SlowJoin& j, uint32_t* out) {
    if (j.st != LYON_OK || j.vcount >= (1u << 21) || j.from_neg_rel > 3u || j.from_pos_rel > 3u ||
        (j.to_f & ~EF_SELF_EQ) != 0 || j.jtris + 4u < j.vcount || j.jtris + 4u - j.vcount > 7u)
        return false;
    *out = j.vcount | (j.from_neg_rel << 21) | (j.from_pos_rel << 23) |
           ((j.jtris + 4u - j.vcount) << 25) | (j.to_f ? 1u << 28 : 0u);
    return true;
}
__device__ __forceinline__ uint32_t pj_vertices(uint32_t j) { return j & 0x1FFFFFu; }
__device__ __forceinline__ uint32_t pj_neg(uint32_t j) { return (j >> 21) & 3u; }
__device__ __forceinline__ uint32_t pj_pos(uint32_t j) { return (j >> 23) & 3u; }
__device__ __forceinline__ uint32_t pj_tris(uint32_t j) {
    return pj_vertices(j) + ((j >> 25) & 7u) - 4u;
}
__device__ __forceinline__ uint32_t pj_to(uint32_t j) { return (j >> 28) & 1u ? EF_SELF_EQ : 0u; }
__device__ __forceinline__ uint32_t pj_from(uint32_t j) {
    return pj_neg(j) == pj_pos(j) ? EF_SELF_EQ : 0u;
}

// A flattening step's join, packed.
constexpr uint32_t PACKED_STEP = 2u | (1u << 21) | (2u << 25);

// ---- a verb's curve units ---------------------------------------------------------------------
// Its first point, and the point before its last one (`from` when it is one step).
__device__ __forceinline__ V2 first_point(const Unit& u) {
    return u.m >= 2 ? poly_sample(u.p, u.t0 + u.s) : u.to;
}
__device__ __forceinline__ V2 point_before_end(const Unit& u, V2 from) {
    return u.m >= 2 ? poly_sample(u.p, unit_t(u, u.m - 1)) : from;
}

// The one or two units of a segment verb, with lyon's arithmetic (setup_verb, stroke_parts.cuh).
// `cut`: the parameter of a sharp turn (VF_TURN), or for a verb that is cut (VF_CUT) the step of
// the join between its runs and, in the upper 16 bits, how many steps merge into that point.
__device__ __forceinline__ void verb_units(int kind, uint32_t p, const float* points, float tol,
                                           uint32_t flags, uint32_t cut, Unit& a, Unit& b) {
    b.m = 0;
    if (kind == LYON_VERB_LINE_TO) {
        a.to = load_pt(points, p);
        a.m = 1;
        a.s = 1.0f;
        a.t0 = 0.0f;
        return;
    }
    const V2 from = load_pt(points, p - 1);
    if (kind == LYON_VERB_QUADRATIC_TO) {
        const V2 ctrl = load_pt(points, p), to = load_pt(points, p + 1);
        if (flags & VF_TURN) {
            const float ts = __uint_as_float(cut);
            const V2 sp = quad_sample(from, ctrl, to, ts);
            const V2 bc = lerp(from, ctrl, ts), ac = lerp(ctrl, to, ts);
            unit_of(a, quad_poly(from, bc, sp), sp, quad_wang(from, bc, sp, tol));
            unit_of(b, quad_poly(sp, ac, to), to, quad_wang(sp, ac, to, tol));
            return;
        }
        unit_of(a, quad_poly(from, ctrl, to), to, quad_wang(from, ctrl, to, tol));
    } else {
        const V2 c1 = load_pt(points, p), c2 = load_pt(points, p + 1), to = load_pt(points, p + 2);
        unit_of(a, cubic_poly(from, c1, c2, to), to, cubic_wang(from, c1, c2, to, tol));
    }
    if (flags & VF_CUT) {
        const uint32_t at = cut & 0xFFFFu, gap = cut >> 16;
        const float t = unit_t(a, at);
        b = a;
        b.m = a.m - at - gap;
        b.t0 = accumulate_t(a.s, at, t, at + gap);
        a.m = at;
        a.to = poly_sample(a.p, t);
    }
}

// The end point of the verb in `slot` (a Begin or a segment).
__device__ __forceinline__ V2 end_point(const StrokeVerbs& S, const float* points, uint32_t slot) {
    const int k = S.kind[slot] & KIND_MASK;
    return load_pt(points, S.rec[slot] + points_of_verb(k) - 1);
}
// Its last kept point, once walk_kernel has run: the end point, or the step it merged into.
__device__ __forceinline__ V2 last_kept(const StrokeVerbs& S, const float* points, uint32_t slot) {
    const int k = S.kind[slot] & KIND_MASK;
    if (k != LYON_VERB_BEGIN && (S.flags[slot] & VF_MERGED)) {
        const float2 f = S.fin[slot];
        return V2{f.x, f.y};
    }
    return load_pt(points, S.rec[slot] + points_of_verb(k) - 1);
}

__device__ __forceinline__ void leave_to_walk(const StrokeVerbs& S, uint32_t path) {
    S.path_walk[path] = 1u;
}

__device__ __forceinline__ uint32_t batch_verbs(const StrokeArgs& A) {
    const uint32_t a = A.verb_offsets[0], b = A.verb_offsets[A.num_paths];
    return b >= a ? b - a : 0u;
}

// Slots per tile of a grid whose blocks take tiles in turn: `most`, or fewer (at least `least`) when
// that would leave blocks without a tile.
__device__ __forceinline__ uint32_t tile_size(uint32_t nv, uint32_t least, uint32_t most) {
    return min(most, max(least, (nv + gridDim.x - 1u) / gridDim.x));
}

// Whether the count phase has nothing to work on after prepare_kernel: more verbs than the arrays
// hold, or offsets that run backwards (prepare_kernel does not write the slots of such a path, and
// two paths may have written one slot, so nothing in the slots may be followed). The caller takes
// the batch path by path.
__device__ __forceinline__ bool unfit(const StrokeVerbs& S, uint32_t verbs) {
    return verbs > S.cap || S.words[STROKE_VERBS_UNFIT] != 0;
}

}  // namespace
}  // namespace lg
