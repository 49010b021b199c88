// stroke_seq.cu — lyon's sequential stroke stepper, one path per thread.
//
// The warp-per-path kernel (stroke.cu) reproduces the fixed-width stroker's output without
// running its state machine step by step. Two outputs need the state machine itself:
//   * variable line width (StrokeOptions::variable_line_width, stroke.rs:654-767): every edge's
//     side attachments depend on both endpoints' widths (step_impl, stroke.rs:1380-1512);
//   * vertex sources (StrokeVertex::source, stroke.rs:2719-2722): every vertex carries the
//     VertexSource of the join, cap or edge it was made for, and custom attributes are
//     interpolated from those (StrokeVertex::interpolated_attributes, stroke.rs:2728-2747).
// Here one thread walks a path's events as tessellate_with_ids_fw/_vw do (stroke.rs:654-870):
// each endpoint or flattened curve point is stepped with fixed_width_step_impl
// (stroke.rs:1521-1632) or step_impl, and the sub-path ends with end/close/end_with_caps
// (stroke.rs:1179-1378). The sources of the points in the stepper's three-point buffer and of
// its `firsts` are kept beside them, so every emitted vertex gets its source the way lyon's
// `self.vertex.src` does. Both passes (count and emit) run this walk, so their counts agree by
// construction.
#include "stroke_core.cuh"
#include "stroke_out.cuh"
#include "stroke_seq.cuh"
#include "kernels.h"

namespace lg {

namespace {

constexpr uint32_t FULL = 0xFFFFFFFFu;

// A flattened run of a curve: lyon's for_each_flattened_with_t loop (quadratic_bezier.rs:891-938,
// cubic_bezier.rs:1318-1363: t advances by 1/n, the last point is the end point at t = 1), with
// the curve parameter mapped to the whole curve as flatten_quad does for a split quadratic
// (stroke.rs:2755-2779: t = tadd + t_run * tmul). That t gives the point's source and, with a
// variable width, its half width (linear in t between the endpoints' widths, stroke.rs:1022,
// 1060).
template <bool VW, class SK>
__device__ __noinline__ void seq_flatten(Stepper<VW>& stepper, Keep& keep, const Poly& poly, V2 to,
                                         float n, float tmul, float tadd, float sw, float ew,
                                         uint32_t from_id, uint32_t to_id, const StrokeParams& P,
                                         SK& sink, int* status) {
    Stepper<VW> T = stepper;
    SK s = sink;
    const Poly pl = poly;
    const StrokeParams p = P;
    int st = *status;
    const float step = 1.0f / n;
    const uint32_t count = to_u32_or1(n) - 1;
    float t0 = 0.0f;
    for (uint32_t i = 0; i <= count; ++i) {
        const bool last = i == count;
        const float t1 = last ? 1.0f : t0 + step;
        const V2 q = last ? to : poly_sample(pl, t1);
        const float t = tadd + t1 * tmul;
        stepper_step<VW, true>(T, q, VW ? (sw * (1.0f - t) + ew * t) * 0.5f : p.hw, t1 != 1.0f,
                               __int_as_float(0x7fc00000), curve_src(from_id, to_id, t), p, s, st,
                               &keep);
        t0 = t1;
    }
    stepper = T;
    sink = s;
    *status = st;
}

// One thread strokes one path (tessellate_with_ids_fw / _vw, stroke.rs:654-870). With a variable
// width an endpoint's half width is line_width x its factor x 0.5. Endpoint ids are the points'
// indices in the batch. Verbs are checked as they come (a Begin inside a sub-path, a sub-path
// without Begin, missing points or an unknown verb fail the path with
// LYON_ERR_INVALID_ARGUMENT).
template <bool EMIT, bool VW, class SK>
__device__ __noinline__ void stroke_path_sequential(const StrokeArgs& A, uint32_t path) {
    const PathOut po = path_out<EMIT, SK::kRec>(A, path);
    const uint32_t v_begin = A.verb_offsets[path], v_end = A.verb_offsets[path + 1];
    const uint32_t p_end = A.point_offsets[path + 1];
    const lyon_stroke_options opt = A.options[A.num_options > 1 ? path : 0];
    const StrokeParams P = make_params(opt);
    const float lw = opt.line_width;
    const size_t ws = A.width_stride ? A.width_stride : 1u;
    SK s;
    s.id_base = po.id_base;
    s.nv = 0;
    s.ni = 0;
    s.vout = po.vout;
    s.rout = po.rout;
    s.iout = po.iout;
    s.index_bits = po.bits;
    s.vcap = po.vmax;
    s.icap = po.imax;
    s.overflow = false;
    s.adv = 0.0f;
    if (EMIT) set_sout(s, A.sources + A.vtx_offsets[path]);
    set_src(s, endpoint_src(LYON_NO_ENDPOINT));
    Stepper<VW> S;
    stepper_init(S);
    Keep keep;
    keep.nfirsts = 0;
    keep.mnec = false;
    float start_adv = 0.0f;  // sub_path_start_advancement
    int status = LYON_OK;
    bool open = false;
    V2 cur = V2{0.0f, 0.0f};
    float cur_w = 1.0f;
    uint32_t cur_id = 0;
    uint32_t pc = A.point_offsets[path];
    for (uint32_t vi = v_begin; vi < v_end && status == LYON_OK; ++vi) {
        const int k = A.verbs[vi];
        if (k > LYON_VERB_END || pc + points_of_verb(k) > p_end ||
            (k == LYON_VERB_BEGIN) == open) {
            status = LYON_ERR_INVALID_ARGUMENT;
            break;
        }
        if (k == LYON_VERB_BEGIN || k == LYON_VERB_LINE_TO) {
            cur = load_pt(A.points, pc);
            if (VW) cur_w = A.widths[pc * ws];
            cur_id = pc;
            ++pc;
            float adv = __int_as_float(0x7fc00000);
            if (k == LYON_VERB_BEGIN) {
                open = true;
                keep.mnec = false;
                adv = start_adv;
            }
            stepper_step<VW, true>(S, cur, VW ? lw * cur_w * 0.5f : P.hw, false, adv,
                                   endpoint_src(cur_id), P, s, status, &keep);
        } else if (k == LYON_VERB_QUADRATIC_TO) {
            const V2 ctrl = load_pt(A.points, pc);
            const V2 to = load_pt(A.points, pc + 1);
            const uint32_t to_id = pc + 1;
            const float w1 = VW ? A.widths[(pc + 1) * ws] : 1.0f;
            pc += 2;
            const float sw = lw * cur_w, ew = lw * w1;
            float ts;
            if (find_sharp_turn(cur, ctrl, to, &ts)) {
                const V2 sp = quad_sample(cur, ctrl, to, ts);
                const V2 bc = lerp(cur, ctrl, ts);
                const V2 ac = lerp(ctrl, to, ts);
                seq_flatten<VW>(S, keep, quad_poly(cur, bc, sp), sp, quad_wang(cur, bc, sp, P.tolerance),
                                ts, 0.0f, sw, ew, cur_id, to_id, P, s, &status);
                seq_flatten<VW>(S, keep, quad_poly(sp, ac, to), to, quad_wang(sp, ac, to, P.tolerance),
                                1.0f - ts, ts, sw, ew, cur_id, to_id, P, s, &status);
            } else {
                seq_flatten<VW>(S, keep, quad_poly(cur, ctrl, to), to,
                                quad_wang(cur, ctrl, to, P.tolerance), 1.0f, 0.0f, sw, ew, cur_id,
                                to_id, P, s, &status);
            }
            cur = to;
            cur_w = w1;
            cur_id = to_id;
        } else if (k == LYON_VERB_CUBIC_TO) {
            const V2 c1 = load_pt(A.points, pc);
            const V2 c2 = load_pt(A.points, pc + 1);
            const V2 to = load_pt(A.points, pc + 2);
            const uint32_t to_id = pc + 2;
            const float w1 = VW ? A.widths[(pc + 2) * ws] : 1.0f;
            pc += 3;
            seq_flatten<VW>(S, keep, cubic_poly(cur, c1, c2, to), to,
                            cubic_wang(cur, c1, c2, to, P.tolerance), 1.0f, 0.0f, lw * cur_w,
                            lw * w1, cur_id, to_id, P, s, &status);
            cur = to;
            cur_w = w1;
            cur_id = to_id;
        } else {  // Close or End
            if (k == LYON_VERB_CLOSE) ++pc;
            stepper_end<VW>(S, keep, k == LYON_VERB_CLOSE, P, s, &status, &start_adv);
            stepper_init(S);
            keep.nfirsts = 0;
            open = false;
        }
    }
    if (s.overflow && status == LYON_OK) status = LYON_ERR_INTERNAL;
    finish_path<EMIT>(A, path, s.nv, s.ni, status, po);
}

// 32 paths per warp, one per lane, from the launch's work counter.
template <bool EMIT, bool VW, class SK>
__global__ void __launch_bounds__(256) stroke_seq_kernel(StrokeArgs A) {
    const int lane = threadIdx.x & 31;
    const uint32_t n = A.list_only ? min(*A.item_split, A.num_paths) : A.num_paths;
    for (;;) {
        uint32_t first = 0;
        if (lane == 0) first = atomicAdd(A.work_counter, 32u);
        first = __shfl_sync(FULL, first, 0);
        if (first >= n) break;
        const uint32_t item = first + (uint32_t)lane;
        if (item < n) {
            const uint32_t path = A.list_only ? A.order[item] : item;
            if (!EMIT || A.status[path] == LYON_OK) stroke_path_sequential<EMIT, VW, SK>(A, path);
        }
        __syncwarp();
    }
}

template <bool VW>
void launch_seq(const StrokeArgs& a, bool emit, int grid, cudaStream_t s) {
    if (!emit) {
        stroke_seq_kernel<false, VW, Sink><<<grid, 256, 0, s>>>(a);
    } else if (a.sources && a.vertex_attrs) {
        stroke_seq_kernel<true, VW, SrcSinkT<true>><<<grid, 256, 0, s>>>(a);
    } else if (a.sources) {
        stroke_seq_kernel<true, VW, SrcSinkT<false>><<<grid, 256, 0, s>>>(a);
    } else if (a.vertex_attrs) {
        stroke_seq_kernel<true, VW, RecSink><<<grid, 256, 0, s>>>(a);
    } else {
        stroke_seq_kernel<true, VW, Sink><<<grid, 256, 0, s>>>(a);
    }
}

}  // namespace

cudaError_t launch_stroke_seq(const StrokeArgs& args, bool emit, int grid, cudaStream_t stream) {
    if (args.widths) {
        launch_seq<true>(args, emit, grid, stream);
    } else {
        launch_seq<false>(args, emit, grid, stream);
    }
    note_launches(1);
    return cudaGetLastError();
}

}  // namespace lg
