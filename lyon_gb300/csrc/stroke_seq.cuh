// stroke_seq.cuh — lyon's sequential stroke stepper with vertex sources: one step of a point, and
// the end of a sub-path (used by the path-per-thread kernels of stroke_seq.cu and the
// verb-per-thread kernels of stroke_steps.cu).
#pragma once

#include "stroke_core.cuh"
#include "stroke_out.cuh"

namespace lg {
namespace {

__device__ __forceinline__ lyon_vertex_source endpoint_src(uint32_t id) {
    return lyon_vertex_source{id, LYON_NO_ENDPOINT, 0.0f};
}

// A point at parameter t of the curve between two endpoints; at t == 1 the end point itself
// (stroke.rs:1007-1016, 1045-1053, 1119-1128, 1154-1163).
__device__ __forceinline__ lyon_vertex_source curve_src(uint32_t from, uint32_t to, float t) {
    return t == 1.0f ? endpoint_src(to) : lyon_vertex_source{from, to, t};
}

// A sink that also writes every vertex's source: `src` is set by the stepper before each group
// of vertices, as `adv` is.
template <bool REC>
struct SrcSinkT : SinkT<REC> {
    static constexpr bool kSrc = true;
    lyon_vertex_source* sout;
    lyon_vertex_source src;
    __device__ __forceinline__ uint32_t vertex(V2 p, V2 n, int side) {
        if (this->nv < this->vcap) sout[this->nv] = src;
        return SinkT<REC>::vertex(p, n, side);
    }
};

template <class SK>
__device__ __forceinline__ void set_src(SK&, const lyon_vertex_source&) {}
template <bool REC>
__device__ __forceinline__ void set_src(SrcSinkT<REC>& s, const lyon_vertex_source& v) {
    s.src = v;
}
template <class SK>
__device__ __forceinline__ void set_sout(SK&, lyon_vertex_source*) {}
template <bool REC>
__device__ __forceinline__ void set_sout(SrcSinkT<REC>& s, lyon_vertex_source* p) {
    s.sout = p;
}

// The stepper's state (point buffer, firsts, may_need_empty_cap, sub_path_start_advancement)
// and the sources of the buffered points, slot for slot.
struct SeqStroker {
    VwState W;
    lyon_vertex_source src[3];
    lyon_vertex_source first_src[2];
};

__device__ __forceinline__ uint32_t slot_last(const SeqBuffer& pb) {
    return (pb.start + pb.count - 1) % 3;
}
__device__ __forceinline__ uint32_t slot_second_last(const SeqBuffer& pb) {
    return (pb.start + pb.count - 2) % 3;
}

// One step (fixed_width_step_impl or step_impl) of a point whose source is `src`. The vertices
// the step emits belong to the join at the buffer's last point, so they take its source. Without
// a source-writing sink the bookkeeping compiles away.
template <bool VW, class SK>
__device__ __forceinline__ bool seq_step_any(SeqStroker& S, const DEP& next,
                                             lyon_vertex_source src, const StrokeParams& P,
                                             SK& sink, int* status) {
    VwState& W = S.W;
    SeqBuffer& pb = W.pb;
    const uint32_t count0 = pb.count, start0 = pb.start, n0 = pb.n, nfirsts0 = W.nfirsts;
    if constexpr (SK::kSrc) {
        if (count0 > 0) set_src(sink, S.src[slot_last(pb)]);
    }
    bool ok;
    if constexpr (VW) {
        ok = vw_step(W, next, P, sink, status);
    } else {
        ok = seq_step(pb, next, P, sink, &W.mnec, status);
        // The first join records the sub-path's first two points (stroke.rs:1624-1627).
        if (ok && count0 == 2) {
            W.firsts[0] = pb.pts[0];
            W.firsts[1] = pb.pts[1];
            W.nfirsts = 2;
        }
    }
    if (!ok) return false;
    if constexpr (SK::kSrc) {
        if (nfirsts0 < 2 && W.nfirsts == 2) {
            S.first_src[0] = S.src[0];
            S.first_src[1] = S.src[1];
        }
        if (pb.n > n0) {
            S.src[count0 < 3 ? count0 : start0] = src;  // SeqBuffer::push
        } else {
            S.src[slot_last(pb)] = src;  // SeqBuffer::replace_last (a skipped flattening step)
        }
    }
    return true;
}

// end (stroke.rs:1179-1193) with close (1206-1279), end_with_caps (1322-1378) and the empty cap
// (1282-1316), on the stepper's own points.
template <bool VW, class SK>
__device__ __noinline__ void seq_end(SeqStroker& S, bool close, const StrokeParams& P, SK& sink,
                                     int* status) {
    VwState& W = S.W;
    SeqBuffer& pb = W.pb;
    const uint32_t count = pb.count;
    W.mnec |= close && count == 1;
    if (close && count > 2) {
        DEP p = W.firsts[0];
        const float start_adv = p.adv;
        p.adv = __int_as_float(0x7fc00000);
        const lyon_vertex_source s0 = S.first_src[0], s1 = S.first_src[1];
        if (!seq_step_any<VW>(S, p, s0, P, sink, status)) pb.last().pos = p.pos;
        if (W.nfirsts >= 2) {
            seq_step_any<VW>(S, W.firsts[1], s1, P, sink, status);
            DEP& p0 = pb.second_last();
            DEP& p1 = pb.last();
            sink.adv = start_adv;
            set_src(sink, S.src[slot_second_last(pb)]);
            for (int side = 0; side < 2; ++side) {
                const V2 sp = p0.s[side].has_single ? p0.s[side].single : p0.s[side].next;
                const V2 normal = (sp - p0.pos) / p0.hw;
                p0.s[side].next_vertex = sink.vertex(p0.pos + normal * p0.hw, normal, side);
            }
            add_edge_triangles(p0, p1, sink);
        }
    } else if (W.mnec && count == 1) {
        const DEP& point = pb.first();
        sink.adv = point.adv;
        set_src(sink, S.src[pb.start % 3]);
        if (P.start_cap == LYON_CAP_SQUARE) {
            tessellate_empty_square_cap(point.pos, point.hw, sink);
        } else if (P.start_cap == LYON_CAP_ROUND) {
            tessellate_empty_round_cap(point.pos, point.hw, P, sink, status);
        }
    } else if (count >= 2) {
        DEP p0 = pb.second_last();
        DEP p1 = pb.last();
        if (!VW) {
            // With a fixed width only the joins have side points so far (stroke.rs:1338-1346).
            const V2 tan = normalize(p1.pos - p0.pos);
            const V2 n = V2{-tan.y, tan.x} * p1.hw;
            p1.s[SP].prev = p1.pos + n;
            p1.s[SN].prev = p1.pos - n;
        }
        // tessellate_last_edge sets the last point's advancement (stroke.rs:2140), which the
        // next sub-path starts from.
        p1.adv = p0.adv + vlength(p1.pos - p0.pos);
        set_src(sink, S.src[slot_last(pb)]);
        tessellate_last_edge(p0, p1, count == 2, P, sink, status);
        W.start_adv = p1.adv;
        lyon_vertex_source fs = S.src[slot_second_last(pb)];
        if (count > 2) {
            p0 = W.firsts[0];
            p1 = W.firsts[1];
            fs = S.first_src[0];
        }
        set_src(sink, fs);
        tessellate_first_edge(p0, p1, P, sink, status);
    }
    pb.start = pb.count = pb.n = 0;
    W.nfirsts = 0;
}

// ---- the stepper in registers ------------------------------------------------------------------
// seq_step_any over three points in local memory takes about 2 us a step, nearly all of it loads
// and stores of the points. All that later steps read of the last two points is here; the rest
// (the joins in full) is only kept for the sub-path's first two points and its end.
template <bool VW>
struct Stepper {
    uint32_t count;  // points, at most 3
    // The second last point: sides towards the last one, ids an edge from it starts with.
    V2 ppos, pnext_p, pnext_n;
    float phw, padv;
    uint32_t pneg, ppid;
    bool pgen;  // its join was a general one (Keep::join holds it)
    // The last point: sides from the second last one (variable width).
    V2 lpos, lprev_p, lprev_n;
    float lhw, ladv;
    bool lflat;
    lyon_vertex_source psrc, lsrc;
};

// What the end of a sub-path needs besides: lyon's firsts, and the last general join.
struct Keep {
    DEP first[2], join;
    lyon_vertex_source first_src;
    uint32_t nfirsts;
    bool mnec;
};

template <bool VW>
__device__ __forceinline__ void stepper_init(Stepper<VW>& T) {
    const V2 nan = V2{__int_as_float(0x7fc00000), __int_as_float(0x7fc00000)};
    T.count = 0;
    T.ppos = T.lpos = V2{0.0f, 0.0f};
    T.pnext_p = T.pnext_n = T.lprev_p = T.lprev_n = nan;
    T.phw = T.lhw = T.padv = T.ladv = 0.0f;
    T.pneg = T.ppid = INVALID_ID;
    T.pgen = T.lflat = false;
    T.psrc = T.lsrc = endpoint_src(LYON_NO_ENDPOINT);
}

// Side points of an edge's two ends and its length (vw_edge_attachments).
struct EdgeSides {
    V2 next_p, next_n, prev_p, prev_n;
    float d;
};
static __device__ __noinline__ EdgeSides edge_sides_vw(V2 p0, float hw0, V2 p1, float hw1) {
    DEP a, b;
    dep_init(a, p0, hw0, LYON_JOIN_MITER, false);
    dep_init(b, p1, hw1, LYON_JOIN_MITER, false);
    a.adv = 0.0f;
    vw_edge_attachments(a, b);
    return EdgeSides{a.s[SP].next, a.s[SN].next, b.s[SP].prev, b.s[SN].prev, b.adv};
}

// A join that is no flattening step, with its edge and triangles.
template <class SK>
struct GeneralOut {
    SK sink;
    V2 next_p, next_n;
    uint32_t neg, pid;
    int st;
};
template <bool VW, class SK>
__device__ __noinline__ GeneralOut<SK> general_step(Stepper<VW> T, V2 lnext_p, V2 lnext_n, V2 pos,
                                                    V2 nprev_p, V2 nprev_n, float nadv,
                                                    StrokeParams P, SK s, DEP* keep) {
    DEP J;
    dep_init(J, T.lpos, T.lhw, P.line_join, T.lflat);
    J.adv = T.ladv;
    int st = LYON_OK;
    if constexpr (VW) {
        DEP prev, next;
        dep_init(prev, T.ppos, T.phw, P.line_join, false);
        prev.adv = T.padv;
        prev.s[SP].next = T.pnext_p;
        prev.s[SN].next = T.pnext_n;
        dep_init(next, pos, T.lhw, P.line_join, false);
        next.adv = nadv;
        next.s[SP].prev = nprev_p;
        next.s[SN].prev = nprev_n;
        J.s[SP].prev = T.lprev_p;
        J.s[SN].prev = T.lprev_n;
        J.s[SP].next = lnext_p;
        J.s[SN].next = lnext_n;
        vw_join_sides(prev, J, next, P.miter_limit, SP);
        vw_join_sides(prev, J, next, P.miter_limit, SN);
        // Prevent folding when the other side is concave.
        if (J.s[SP].has_single) J.fold[SN] = false;
        if (J.s[SN].has_single) J.fold[SP] = false;
    } else {
        compute_join_side_positions_fw(T.ppos, J, pos, P.miter_limit);
    }
    add_join_base_vertices(J, SN, s);
    add_join_base_vertices(J, SP, s);
    uint32_t neg, pid;
    if (T.count > 2) {
        edge_ids_to(J, &neg, &pid);
        edge_triangles(T.pneg, T.ppid, neg, pid, &s);
    }
    tessellate_join(J, P, s, &st);
    edge_ids_from(J, &neg, &pid);
    if (keep) *keep = J;
    return GeneralOut<SK>{s, J.s[SP].next, J.s[SN].next, neg, pid, st};
}

// A flattening step's join as lyon's EndpointData, from the stepper's second last point.
template <bool VW>
__device__ __forceinline__ void step_dep(DEP& d, const Stepper<VW>& T) {
    fast_join_dep(d, T.ppos, T.phw, T.pnext_p, T.pnext_n, T.ppid, T.pneg);
    d.adv = T.padv;
}

// One step: seq_step_any's, in registers. With KEEP the sub-path's firsts, its merges into the
// first point and the last general join go to `keep`.
template <bool VW, bool KEEP, class SK>
__device__ __forceinline__ void stepper_step(Stepper<VW>& T, V2 pos, float hw, bool flat, float adv,
                                             lyon_vertex_source src, const StrokeParams& P,
                                             SK& sink, int& status, Keep* keep) {
    constexpr bool ADV = VW || SK::kRec;
    if (T.count > 0 && too_close(T.lpos, pos, P.merge_threshold)) {
        if (KEEP && T.count == 1) keep->mnec = true;
        return;
    }
    const V2 nan = V2{__int_as_float(0x7fc00000), __int_as_float(0x7fc00000)};
    V2 next_p = nan, next_n = nan, prev_p = nan, prev_n = nan;  // sides of the edge to `pos`
    const V2 ne = pos - T.lpos;
    if constexpr (VW) {
        if (T.count > 0 && (!T.lflat || !flat)) {
            const EdgeSides e = edge_sides_vw(T.lpos, T.lhw, pos, hw);
            next_p = e.next_p;
            next_n = e.next_n;
            prev_p = e.prev_p;
            prev_n = e.prev_n;
            if (isnan(adv)) adv = T.ladv + e.d;
        }
    } else if (T.count == 1) {
        const V2 tan = ne / vlength(ne);
        const V2 n = V2{-tan.y, tan.x} * hw;
        next_p = T.lpos + n;
        next_n = T.lpos - n;
        if (ADV && isnan(adv)) adv = T.ladv + vlength(ne);
    }
    uint32_t neg = INVALID_ID, pid = INVALID_ID;
    bool general = false;
    if (T.count > 1) {
        set_src(sink, T.lsrc);
        const V2 pe = T.lpos - T.ppos;
        if (!VW && ADV && isnan(T.ladv)) T.ladv = T.padv + vlength(pe);
        if (T.lflat && dot(pe, ne) > 0.0f) {
            // flattened_step (stroke.rs:1743-1806)
            const float pl = vlength(pe), nl = vlength(ne);
            if (VW && isnan(T.ladv)) T.ladv = T.padv + pl;
            if (ADV && isnan(adv)) adv = T.ladv + nl;
            sink.adv = T.ladv;
            const V2 normal = compute_normal(pe / pl, ne / nl);
            next_p = T.lpos + normal * T.lhw;
            next_n = T.lpos - normal * T.lhw;
            const bool skip = dot(pe, next_p - T.pnext_p) < 0.0f &&
                              dot(pe, next_n - T.pnext_n) < 0.0f;
            if (VW && skip) {
                // The point before is replaced by this one.
                T.lpos = pos;
                T.lprev_p = prev_p;
                T.lprev_n = prev_n;
                T.lhw = hw;
                T.ladv = adv;
                T.lflat = flat;
                T.lsrc = src;
                return;
            }
            if (!skip) {
                pid = sink.vertex(next_p, normal, SP);
                neg = sink.vertex(T.lpos + (-normal) * T.lhw, -normal, SN);
            }
            if (T.count > 2) edge_triangles(T.pneg, T.ppid, neg, pid, &sink);
        } else {
            sink.adv = T.ladv;
            general = true;
            const GeneralOut<SK> g = general_step<VW>(T, next_p, next_n, pos, prev_p, prev_n, adv, P,
                                                      sink, KEEP ? &keep->join : nullptr);
            sink = g.sink;
            next_p = g.next_p;
            next_n = g.next_n;
            neg = g.neg;
            pid = g.pid;
            if (g.st != LYON_OK) status = g.st;
        }
        if (KEEP && T.count == 2) {
            DEP& f = keep->first[0];
            dep_init(f, T.ppos, T.phw, P.line_join, false);
            f.adv = T.padv;
            f.s[SP].next = T.pnext_p;
            f.s[SN].next = T.pnext_n;
            keep->first_src = T.psrc;
        }
    }
    // Push.
    const bool first_join = T.count == 2;
    T.ppos = T.lpos;
    T.pnext_p = next_p;
    T.pnext_n = next_n;
    T.phw = T.lhw;
    T.padv = T.ladv;
    T.pneg = neg;
    T.ppid = pid;
    T.pgen = general;
    T.psrc = T.lsrc;
    T.lpos = pos;
    T.lprev_p = prev_p;
    T.lprev_n = prev_n;
    T.lhw = hw;
    T.ladv = adv;
    T.lflat = flat;
    T.lsrc = src;
    if (T.count < 3) ++T.count;
    if (KEEP && first_join) {
        if (general) {
            keep->first[1] = keep->join;
        } else {
            step_dep(keep->first[1], T);
        }
        keep->nfirsts = 2;
    }
}

// The end of the sub-path (seq_end) from the stepper's state.
template <bool VW, class SK>
__device__ __noinline__ void stepper_end(const Stepper<VW>& T, const Keep& K, bool close,
                                         const StrokeParams& P, SK& sink, int* status,
                                         float* start_adv) {
    SeqStroker S;
    SeqBuffer& pb = S.W.pb;
    pb.start = 0;
    pb.count = pb.n = T.count;
    S.W.mnec = K.mnec;
    S.W.nfirsts = K.nfirsts;
    S.W.start_adv = *start_adv;
    if (K.nfirsts == 2) {
        S.W.firsts[0] = K.first[0];
        S.W.firsts[1] = K.first[1];
        S.first_src[0] = K.first_src;
        S.first_src[1] = T.psrc;  // read by no vertex
    }
    if (T.count > 0) {
        const uint32_t l = T.count - 1;
        dep_init(pb.pts[l], T.lpos, T.lhw, P.line_join, T.lflat);
        pb.pts[l].adv = T.ladv;
        pb.pts[l].s[SP].prev = T.lprev_p;
        pb.pts[l].s[SN].prev = T.lprev_n;
        S.src[l] = T.lsrc;
        if (l > 0) {
            DEP& d = pb.pts[l - 1];
            if (T.count == 2) {
                dep_init(d, T.ppos, T.phw, P.line_join, false);
                d.adv = T.padv;
                d.s[SP].next = T.pnext_p;
                d.s[SN].next = T.pnext_n;
            } else if (T.pgen) {
                d = K.join;
            } else {
                step_dep(d, T);
            }
            S.src[l - 1] = T.psrc;
        }
    }
    seq_end<VW>(S, close, P, sink, status);
    *start_adv = S.W.start_adv;
}

}  // namespace
}  // namespace lg
