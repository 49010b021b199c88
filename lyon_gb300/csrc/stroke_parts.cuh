// stroke_parts.cuh — the pieces of the fixed-width stroke that the walk of one path by one warp
// (stroke.cu) and the verb-parallel kernels (stroke_verbs.cu) share: a verb's flattening
// parameters and the tail of a sub-path.
#pragma once

#include "stroke_core.cuh"
#include "stroke_out.cuh"

namespace lg {

constexpr uint32_t MAX_VERB_STEPS = 1u << 26;

struct VerbSlot {
    Poly pA, pB;
    V2 toA, toB;
    float sA, sB;
    uint32_t mA, mB;
    uint32_t excl, steps;  // first step of the verb within the window, step count
    int kind;
};

// Everything the tail of a sub-path needs (stroke.rs:1179-1378): the first three and the last
// three kept points and how their joins were done.
struct TailJob {
    uint32_t path, n, flags, base1, jbase, vcur, icur;
    V2 p0, p1, p2, c3, c2, c1;
    float adv0, adv2, adv1;  // advancements of p0, c2 and c1 (read by the attribute output only)
};
enum : uint32_t {
    TJ_CLOSED = 1u, TJ_MNEC = 2u, TJ_FLAT1 = 4u, TJ_FAST1 = 8u, TJ_SKIP1 = 16u, TJ_F1 = 32u,
    TJ_F2 = 64u, TJ_JFAST = 128u, TJ_JSKIP = 256u
};

// Flattening parameters of one verb of a window (lane = verb): lines and Begin give one step;
// quadratics are split at a sharp turn (stroke.rs:2755-2779, 3178-3212) and each part gets lyon's
// segment count (quadratic_bezier.rs:943-974); cubics likewise (cubic_bezier.rs:1369-1403).
// Returns the number of flattened points the verb contributes and the verb's status (by value,
// so that the caller keeps no status word in local memory).
struct VerbSetup {
    uint32_t steps;
    int st;
};
static __device__ __noinline__ VerbSetup setup_verb(VerbSlot& out, int kind, uint32_t pofs,
                                                    uint32_t pcount, uint32_t p_end,
                                                    const float* points, float tolerance) {
    int vst = LYON_OK;
    VerbSlot sl;
    sl.kind = kind;
    sl.mA = 0;
    sl.mB = 0;
    sl.sA = sl.sB = 0.0f;
    uint32_t steps = 0;
    if (pofs + pcount > p_end || kind < 0) {
        vst = LYON_ERR_INVALID_ARGUMENT;
    } else if (kind == LYON_VERB_BEGIN || kind == LYON_VERB_LINE_TO) {
        sl.toA = load_pt(points, pofs);
        steps = 1;
    } else if (kind == LYON_VERB_QUADRATIC_TO) {
        V2 from = load_pt(points, pofs - 1);
        V2 ctrl = load_pt(points, pofs);
        V2 to = load_pt(points, pofs + 1);
        float ts;
        if (find_sharp_turn(from, ctrl, to, &ts)) {
            V2 sp = quad_sample(from, ctrl, to, ts);
            V2 bc = lerp(from, ctrl, ts);
            V2 ac = lerp(ctrl, to, ts);
            float nA = quad_wang(from, bc, sp, tolerance);
            float nB = quad_wang(sp, ac, to, tolerance);
            sl.pA = quad_poly(from, bc, sp);
            sl.pB = quad_poly(sp, ac, to);
            sl.mA = to_u32_or1(nA);
            sl.mB = to_u32_or1(nB);
            sl.sA = 1.0f / nA;
            sl.sB = 1.0f / nB;
            sl.toA = sp;
            sl.toB = to;
        } else {
            float nA = quad_wang(from, ctrl, to, tolerance);
            sl.pA = quad_poly(from, ctrl, to);
            sl.mA = to_u32_or1(nA);
            sl.sA = 1.0f / nA;
            sl.toA = to;
        }
        steps = sl.mA + sl.mB;
    } else if (kind == LYON_VERB_CUBIC_TO) {
        V2 from = load_pt(points, pofs - 1);
        V2 c1 = load_pt(points, pofs);
        V2 c2 = load_pt(points, pofs + 1);
        V2 to = load_pt(points, pofs + 2);
        float nA = cubic_wang(from, c1, c2, to, tolerance);
        sl.pA = cubic_poly(from, c1, c2, to);
        sl.mA = to_u32_or1(nA);
        sl.sA = 1.0f / nA;
        sl.toA = to;
        steps = sl.mA;
    }
    if (sl.mA > MAX_VERB_STEPS || sl.mB > MAX_VERB_STEPS) {
        vst = LYON_ERR_UNSUPPORTED;
        steps = 0;
    }
    sl.steps = steps;
    sl.excl = 0;
    out = sl;
    return VerbSetup{steps, vst};
}

// A join as lyon's EndpointData after its processing, with vertex ids starting at base_id (the
// fast layout of flattened_step, or the general layout), for firsts[1] and the tail.
static __device__ __noinline__ void join_dep_with_ids(DEP* out, V2 prev, V2 cur, V2 nxt, bool flat,
                                               bool fast, bool skip, uint32_t base_id,
                                               const StrokeParams& P, int* status) {
    if (fast) {
        V2 pe = cur - prev;
        V2 pt = pe / vlength(pe);
        V2 ne = nxt - cur;
        V2 nt = ne / vlength(ne);
        V2 nrm = compute_normal(pt, nt);
        fast_join_dep(*out, cur, P.hw, cur + nrm * P.hw, cur - nrm * P.hw,
                      skip ? INVALID_ID : base_id, skip ? INVALID_ID : base_id + 1);
    } else {
        DEP d = general_join_geometry(prev, cur, flat, nxt, P);
        join_arc_vertices(d, P, status);
        Sink probe{base_id, 0, 0, nullptr, nullptr, 32};
        add_join_base_vertices(d, SN, probe);
        add_join_base_vertices(d, SP, probe);
        *out = d;
    }
}

// Side "next" points of the join at `cur` (neighbours `prev`, `nxt`) when it was a flattening
// step: what the emit pass computed for it (stroke.rs:1760-1776).
struct SidePair {
    V2 pn, nn;
};
static __device__ __noinline__ SidePair fast_join_sides(V2 prev, V2 cur, V2 nxt, float hw) {
    V2 pe = cur - prev;
    V2 pt = pe / vlength(pe);
    V2 ne = nxt - cur;
    V2 nt = ne / vlength(ne);
    V2 nrm = compute_normal(pt, nt);
    return SidePair{cur + nrm * hw, cur - nrm * hw};
}

// The tail of a sub-path: stroke.rs:1179-1279 (end, close) and 1322-1378 (end_with_caps), from
// lyon's firsts (the first kept point with its sides, the first join) and the last join, which
// are rebuilt here from the recorded points. Writes through `s` (positioned at the tail).
template <class SK>
__device__ __noinline__ void run_tail(const TailJob& j, const StrokeParams& P, SK& s,
                                      int* status) {
    const uint32_t n = j.n;
    const bool close = (j.flags & TJ_CLOSED) != 0;
    bool may_need_empty_cap = (j.flags & TJ_MNEC) != 0;
    DEP first0, first1, last;
    dep_init(first0, j.p0, P.hw, P.line_join, false);
    first0.adv = j.adv0;
    if (n >= 2) first_point_sides(first0, j.p1, P.hw);
    if (n >= 3) {
        join_dep_with_ids(&first1, j.p0, j.p1, j.p2, (j.flags & TJ_FLAT1) != 0,
                          (j.flags & TJ_FAST1) != 0, (j.flags & TJ_SKIP1) != 0, j.base1, P,
                          status);
        join_dep_with_ids(&last, j.c3, j.c2, j.c1, (j.flags & TJ_F2) != 0,
                          (j.flags & TJ_JFAST) != 0, (j.flags & TJ_JSKIP) != 0, j.jbase, P,
                          status);
        last.adv = j.adv2;
    }
    const V2 lastp = j.c1;
    const bool lastflat = (j.flags & TJ_F1) != 0;
    may_need_empty_cap |= close && n == 1;
    if (close && n > 2) {
        SeqBuffer pb;
        pb.pts[0] = last;
        dep_init(pb.pts[1], lastp, P.hw, P.line_join, lastflat);
        // The last point's advancement is known to lyon here only when the join before it was
        // a flattening step (stroke.rs:1765-1769); otherwise it is computed again from the
        // point's position, which the merge below may have moved (stroke.rs:1225-1236).
        if (j.flags & TJ_JFAST) pb.pts[1].adv = j.adv1;
        pb.start = 0;
        pb.count = 2;
        pb.n = n;
        bool mnec = false;
        // close (stroke.rs:1206-1279): the first point is stepped again with its advancement
        // recomputed; the two vertices re-made for the first edge keep the starting one.
        DEP p = first0;
        p.adv = __int_as_float(0x7fc00000);
        bool added = seq_step(pb, p, P, s, &mnec, status);
        if (!added) pb.last().pos = p.pos;
        DEP p2 = first1;
        seq_step(pb, p2, P, s, &mnec, status);
        DEP& p0 = pb.second_last();
        DEP& p1 = pb.last();
        s.adv = j.adv0;
        for (int side = 0; side < 2; ++side) {
            V2 sp = p0.s[side].has_single ? p0.s[side].single : p0.s[side].next;
            V2 normal = (sp - p0.pos) / p0.hw;
            p0.s[side].next_vertex = s.vertex(p0.pos + normal * p0.hw, normal, side);
        }
        add_edge_triangles(p0, p1, s);
        return;
    }
    if (may_need_empty_cap && n == 1) {
        V2 pos = first0.pos;
        s.adv = first0.adv;
        if (P.start_cap == LYON_CAP_SQUARE) {
            tessellate_empty_square_cap(pos, P.hw, s);
        } else if (P.start_cap == LYON_CAP_ROUND) {
            tessellate_empty_round_cap(pos, P.hw, P, s, status);
        }
        return;
    }
    if (n >= 2) {
        DEP p0 = (n == 2) ? first0 : last;
        DEP p1;
        dep_init(p1, lastp, P.hw, P.line_join, lastflat);
        p1.adv = j.adv1;
        V2 tan = normalize(p1.pos - p0.pos);
        V2 nn = V2{-tan.y, tan.x} * p1.hw;
        p1.s[SP].prev = p1.pos + nn;
        p1.s[SN].prev = p1.pos - nn;
        tessellate_last_edge(p0, p1, n == 2, P, s, status);
        if (n > 2) {
            p0 = first0;
            p1 = first1;
        }
        tessellate_first_edge(p0, p1, P, s, status);
    }
}

// Runs a tail at the output position (vcur, icur) of its path. Returns the counts it added.
template <bool ATTR>
__device__ __forceinline__ void tail_at(const TailJob& j, const StrokeParams& P,
                                        const PathOut& po, uint32_t* tv, uint32_t* ti,
                                        int* st) {
    SinkT<ATTR> s;
    s.id_base = po.id_base + j.vcur;
    s.nv = 0;
    s.ni = 0;
    s.vout = po.vout ? po.vout + j.vcur : nullptr;
    s.rout = po.rout ? po.rout + j.vcur : nullptr;
    s.iout = nullptr;
    if (po.vout || po.rout) {
        s.iout = po.bits == 16 ? (void*)((uint16_t*)po.iout + j.icur)
                               : (void*)((uint32_t*)po.iout + j.icur);
    }
    s.index_bits = po.bits;
    s.vcap = cap_left(po.vmax, j.vcur);
    s.icap = cap_left(po.imax, j.icur);
    s.overflow = false;
    int tst = LYON_OK;
    run_tail(j, P, s, &tst);
    if (s.overflow && tst == LYON_OK) tst = LYON_ERR_INTERNAL;
    *tv = s.nv;
    *ti = s.ni;
    *st = tst;
}

}  // namespace lg
