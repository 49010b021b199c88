// stroke_verbs.cu — the fixed-width stroke, verb by verb instead of path by path.
//
// lyon's stroker (stroke.rs:1521-1632) steps over the flattened points of a sub-path; the join at
// a point needs that point's two neighbours and nothing else of the state, as long as it is known
// which points the merge filter (stroke.rs:1530-1536) keeps. So every verb can be stroked by
// itself once the kept points around its two ends are known, and a long path is no longer one
// warp's serial work. Count phase:
//   1. prepare_kernel (warp per path) checks the path's grammar, drops the line verbs whose end
//      point the merge filter drops (the only common merges), and packs the rest of the path's
//      verbs into its slots;
//   2. turns_kernel finds the sharp turns at which lyon splits quadratics (f64 sine and cosine:
//      the candidates, a twentieth of a drawing's verbs, are gathered so that full warps do it);
//   3. walk_kernel (lane = flattened point) samples every curve. When each point is kept and each
//      interior join is a flattening step whose skip test cannot fire (the bound of stroke.cu),
//      the verb is regular: its interior is a run of joins of two vertices. With one interior join
//      that is none (a cusp), or a row of steps that merge into one, the verb is cut there into
//      two runs. Anything else is irregular: one
//      thread replays its merge chain. The kept points next to the verb's ends are recorded;
//   4. joins_count_kernel (thread per verb) sizes the general join at each verb's end point from
//      the recorded neighbours, and walks the irregular verbs;
//   5. tails_kernel (thread per sub-path) sizes caps and closings;
//   6. verb_scan_kernel turns the verbs' counts into positions, paths_kernel into path counts; for
//      few paths finish_kernel does what follows the counts, up to the totals, in one launch.
// Emit phase: runs_kernel writes the runs (lane = flattened point), joins_emit_kernel the general
// joins and the irregular verbs, tails_kernel the tails.
//
// A path that breaks the grammar, fails, has a curve of very many steps (of few more than its verbs,
// where one thread would replay them), or may skip a join goes to a list that stroke.cu walks, one
// warp per path, with the status that walk gives. A batch whose offsets run backwards is stroked by
// that walk altogether. Outputs are
// the same bit for bit; tests/test_gpu_stroke_verbs.py compares the two.
//
// Measured, whole calls on one GB300, against the warp-per-path walk for every path: 200,000 curve
// paths (0.47 G vertices) 36.1 -> 8.4 ms, 400,001 map polylines 15.6 -> 1.75 ms, attribute records on
// 20,000 paths 6.4 -> 2.5 ms (by lyon's stepper, a verb per thread, 4.6), 10,000 curve paths
// from and to pinned host memory 9.5 -> 3.6 ms, 1,000 paths of 16 segments 287 -> 250 to 280 us from
// run to run, one such path from and to host arrays 231 -> 155 us. Many short lines are stroked path by
// path (api.cu has the rule and both sides' figures). The walk was bound by the latency of one warp's
// chunks (6,000 to 14,000 cycles for 32 points, its code larger than the instruction cache, the
// longest path last); here no kernel holds more than one stage's code, and parallelism is in verbs
// and points.
#include "scan_core.cuh"
#include "stroke_parts.cuh"
#include "stroke_verbs.cuh"

namespace lg {
namespace {

// The skip test of flattened_step (stroke.rs:1778-1782) cannot fire at a join whose edge into it is
// longer than this bound, when the previous join's side points are symmetric (see stroke.cu).
__device__ __forceinline__ bool skip_impossible(V2 prv, V2 cur, V2 pe, float hw) {
    const float m = fmaxf(fmaxf(fabsf(cur.x), fabsf(cur.y)), fmaxf(fabsf(prv.x), fabsf(prv.y))) +
                    3.0f * hw;
    const float bnd = m * 7.62939453125e-06f;  // 2^-17
    return sqlen(pe) > bnd * bnd;
}

// The skip test itself, at the flattening-step join `cur` after a join at `prv` with side points
// (pn, nn).
__device__ __forceinline__ bool skip_fires(V2 prv, V2 pn, V2 nn, V2 cur, V2 nxt, float hw) {
    const SidePair s = fast_join_sides(prv, cur, nxt, hw);
    const V2 pe = cur - prv;
    return dot(pe, s.pn - pn) < 0.0f && dot(pe, s.nn - nn) < 0.0f;
}

// ---- 1. prepare --------------------------------------------------------------------------------
// One path by one warp, 32 * VPL verbs at a time (VPL to a lane). The windows of a path follow one
// another (points, merges and sub-paths carry over), so a long path is bound by the latency of a
// window: more verbs per window for those, one per lane for the short ones, which are most.
template <int VPL>
__device__ __forceinline__ void prepare_path(const StrokeArgs& A, const StrokeVerbs& S,
                                             uint32_t path, uint32_t v0, uint32_t vb, uint32_t ve,
                                             int lane) {
    uint32_t pc = A.point_offsets[path];
    const uint32_t p_end = A.point_offsets[path + 1];
    const float thr = make_params(A.options[A.num_options > 1 ? path : 0]).merge_threshold;
    const uint32_t slot0 = vb - v0, slot1 = ve - v0;
    uint32_t base = slot0, begin_slot = slot0;
    bool closed = true, bad = false, mnec = false, last_begin = false, gap = false;
    V2 last = V2{0.0f, 0.0f};
    int kinds[VPL];
#pragma unroll
    for (int j = 0; j < VPL; ++j) {
        const uint32_t v = vb + (uint32_t)(lane * VPL + j);
        kinds[j] = v < ve ? (int)A.verbs[v] : 255;
    }
    for (uint32_t vi = vb; vi < ve; vi += 32 * VPL) {
        if constexpr (VPL > 1) {
            // A full window of lines inside a sub-path, none of them short: most of a long
            // polyline. Lane = verb, 32 at a time, so that the loads and stores are in rows.
            bool plain = vi + 32 * VPL <= ve && !closed && !gap && pc + 32 * VPL <= p_end;
#pragma unroll
            for (int j = 0; j < VPL; ++j) plain &= kinds[j] == LYON_VERB_LINE_TO;
            if (__all_sync(FULL, plain)) {
                V2 p[VPL];
#pragma unroll
                for (int j = 0; j < VPL; ++j) p[j] = load_pt(A.points, pc + 32 * j + lane);
                bool close = false;
                V2 left = last;
#pragma unroll
                for (int j = 0; j < VPL; ++j) {
                    V2 q = V2{__shfl_up_sync(FULL, p[j].x, 1), __shfl_up_sync(FULL, p[j].y, 1)};
                    if (lane == 0) q = left;
                    close |= too_close(q, p[j], thr);
                    left = V2{__shfl_sync(FULL, p[j].x, 31), __shfl_sync(FULL, p[j].y, 31)};
                }
                if (!__any_sync(FULL, close)) {
#pragma unroll
                    for (int j = 0; j < VPL; ++j) {
                        const uint32_t slot = base + 32 * j + lane;
                        S.rec[slot] = pc + 32 * j + lane;
                        S.path[slot] = path;
                        S.flags[slot] = 0;
                        S.kind[slot] = (uint8_t)LYON_VERB_LINE_TO;
                        const uint32_t v = vi + (uint32_t)(32 * VPL + lane * VPL + j);
                        kinds[j] = v < ve ? (int)A.verbs[v] : 255;
                    }
                    base += 32 * VPL;
                    pc += 32 * VPL;
                    last = left;
                    last_begin = false;
                    continue;
                }
            }
        }
        int k[VPL];
        uint32_t pofs[VPL], mine = 0;
#pragma unroll
        for (int j = 0; j < VPL; ++j) {
            k[j] = kinds[j];
            // The next window's verbs, loaded a window ahead.
            const uint32_t v = vi + (uint32_t)(32 * VPL + lane * VPL + j);
            kinds[j] = v < ve ? (int)A.verbs[v] : 255;
            pofs[j] = mine;
            mine += points_of_verb(k[j]);
        }
        uint32_t incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t up = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += up;
        }
        // Grammar: a Begin first and after every end, nothing unknown, the points there.
        bool prev_end = __shfl_up_sync(FULL, (int)is_end(k[VPL - 1]), 1) != 0;
        if (lane == 0) prev_end = closed;
        bool wrong = false;
        V2 E[VPL];
#pragma unroll
        for (int j = 0; j < VPL; ++j) {
            pofs[j] += pc + incl - mine;
            if (k[j] == 255 && vi + (uint32_t)(lane * VPL + j) >= ve) continue;
            wrong |= k[j] > LYON_VERB_END || (k[j] == LYON_VERB_BEGIN) != prev_end ||
                     pofs[j] + points_of_verb(k[j]) > p_end;
            prev_end = is_end(k[j]);
        }
        if (__any_sync(FULL, wrong)) {
            bad = true;
            break;
        }
        bool close = false, has_begin = false, has_end = false;
#pragma unroll
        for (int j = 0; j < VPL; ++j) {
            E[j] = V2{0.0f, 0.0f};
            if (k[j] <= LYON_VERB_BEGIN) E[j] = load_pt(A.points, pofs[j] + points_of_verb(k[j]) - 1);
            has_begin |= k[j] == LYON_VERB_BEGIN;
            has_end |= is_end(k[j]);
        }
        const V2 before = V2{__shfl_up_sync(FULL, E[VPL - 1].x, 1),
                             __shfl_up_sync(FULL, E[VPL - 1].y, 1)};
        const bool before_begin = __shfl_up_sync(FULL, (int)(k[VPL - 1] == LYON_VERB_BEGIN), 1) != 0;
        V2 Ep = lane == 0 ? last : before;
#pragma unroll
        for (int j = 0; j < VPL; ++j) {
            close |= k[j] == LYON_VERB_LINE_TO && too_close(Ep, E[j], thr);
            Ep = E[j];
        }
        // The merge chain, replayed for the lanes with a short line step (in order, each from its
        // own predecessor unless the lane before dropped that); elsewhere every verb is kept.
        uint32_t drop = 0, mnecm = 0;  // of this lane's verbs
        const uint32_t begl = __ballot_sync(FULL, has_begin), endl = __ballot_sync(FULL, has_end);
        uint32_t mfirst = 0;  // lanes whose first end closes a sub-path that merged into its Begin
        if (mnec && endl) {
            mfirst = endl & (0u - endl);
            mnec = false;
        }
        uint32_t todo = __ballot_sync(FULL, close);
        int replayed = -2;  // the last replayed lane, what it left and whether it dropped its end
        V2 left = last;
        bool left_begin = false, left_drop = false;
        while (todo) {
            const int l = __ffs(todo) - 1;
            todo &= todo - 1;
            V2 L = before;
            bool one = before_begin, dropped = false, mn = false;
            if (l == 0) {
                L = last;
                one = last_begin;
            } else if (replayed == l - 1 && left_drop) {
                L = left;
                one = left_begin;
            }
            if (lane == l) {
#pragma unroll
                for (int j = 0; j < VPL; ++j) {
                    if (k[j] == 255) continue;
                    dropped = false;
                    if (k[j] == LYON_VERB_BEGIN) {
                        L = E[j];
                        one = true;
                        mn = false;
                    } else if (is_end(k[j])) {
                        if (mn) mnecm |= 1u << j;
                        mn = false;
                    } else if (k[j] == LYON_VERB_LINE_TO && too_close(L, E[j], thr)) {
                        drop |= 1u << j;
                        if (one) mn = true;
                        dropped = true;
                    } else {
                        L = E[j];
                        one = false;
                    }
                }
            }
            left = V2{__shfl_sync(FULL, L.x, l), __shfl_sync(FULL, L.y, l)};
            left_begin = __shfl_sync(FULL, (int)one, l) != 0;
            left_drop = __shfl_sync(FULL, (int)dropped, l) != 0;
            replayed = l;
            if (__shfl_sync(FULL, (int)mn, l) != 0) {
                const uint32_t rest = endl & ~((2u << l) - 1u);
                if (rest) {
                    mfirst |= rest & (0u - rest);
                } else {
                    mnec = true;
                }
            }
            if (left_drop && l < 31) todo |= 2u << l;
        }
        if ((mfirst >> lane) & 1u) {
            bool done = false;
#pragma unroll
            for (int j = 0; j < VPL; ++j) {
                if (!done && is_end(k[j])) {
                    mnecm |= 1u << j;
                    done = true;
                }
            }
        }
        // ---- slots ----
        uint32_t nkeep = 0;
#pragma unroll
        for (int j = 0; j < VPL; ++j) nkeep += k[j] != 255 && !((drop >> j) & 1u) ? 1u : 0u;
        uint32_t kincl = nkeep;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t up = __shfl_up_sync(FULL, kincl, o);
            if (lane >= o) kincl += up;
        }
        // The slot of the last Begin in this lane, and of the one that reigns before the lane.
        uint32_t slot = base + kincl - nkeep, own_begin = 0;
        {
            uint32_t at = slot;
#pragma unroll
            for (int j = 0; j < VPL; ++j) {
                if (k[j] == LYON_VERB_BEGIN) own_begin = at;
                at += k[j] != 255 && !((drop >> j) & 1u) ? 1u : 0u;
            }
        }
        bool gap_j = __shfl_up_sync(FULL, (int)((drop >> (VPL - 1)) & 1u), 1) != 0;
        if (lane == 0) gap_j = gap;
        const uint32_t earlier = begl & ((1u << lane) - 1u);
        uint32_t reign = __shfl_sync(FULL, own_begin, earlier ? 31 - __clz(earlier) : 0);
        if (!earlier) reign = begin_slot;
#pragma unroll
        for (int j = 0; j < VPL; ++j) {
            if (k[j] == 255) continue;
            if ((drop >> j) & 1u) {
                gap_j = true;
                continue;
            }
            if (k[j] == LYON_VERB_BEGIN) reign = slot;
            S.rec[slot] = is_end(k[j]) ? reign : pofs[j];
            S.path[slot] = path;
            S.flags[slot] = 0;
            S.kind[slot] = (uint8_t)(k[j] | ((mnecm >> j) & 1u ? KIND_MNEC : 0u) |
                                     (gap_j ? KIND_GAP : 0u));
            gap_j = false;
            ++slot;
        }
        if (begl) begin_slot = __shfl_sync(FULL, own_begin, 31 - __clz(begl));
        base += __shfl_sync(FULL, kincl, 31);
        pc += __shfl_sync(FULL, incl, 31);
        // The last verb of the window.
        const uint32_t nv = min((uint32_t)(32 * VPL), ve - vi);
        const int ll = (int)((nv - 1) / VPL), lj = (int)((nv - 1) % VPL);
        int lk = 255;
        V2 le = V2{0.0f, 0.0f};
#pragma unroll
        for (int j = 0; j < VPL; ++j)
            if (j == lj) {
                lk = k[j];
                le = E[j];
            }
        lk = __shfl_sync(FULL, lk, ll);
        closed = is_end(lk);
        gap = replayed == ll && left_drop;
        if (gap) {
            last = left;
            last_begin = left_begin;
        } else {
            last = V2{__shfl_sync(FULL, le.x, ll), __shfl_sync(FULL, le.y, ll)};
            last_begin = lk == LYON_VERB_BEGIN;
        }
    }
    if (ve > vb && !closed) bad = true;
    if (lane == 0) S.path_walk[path] = bad ? 1u : 0u;
    __syncwarp();  // a broken path's slots are written again
    for (uint32_t s = (bad ? slot0 : base) + (uint32_t)lane; s < slot1; s += 32)
        S.kind[s] = (uint8_t)KIND_NONE;
}

__global__ void __launch_bounds__(256) prepare_kernel(StrokeArgs A, StrokeVerbs S) {
    const int lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t v0 = A.verb_offsets[0], v1 = A.verb_offsets[A.num_paths];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        S.words[0] = v1 >= v0 ? v1 - v0 : 0u;
        if (v1 < v0) S.words[1] = S.words[STROKE_VERBS_UNFIT] = 1u;
    }
    if (v1 < v0 || v1 - v0 > S.cap) return;
    for (uint32_t path = warp; path < A.num_paths; path += nwarps) {
        const uint32_t vb = A.verb_offsets[path], ve = A.verb_offsets[path + 1];
        if (ve < vb || vb < v0 || ve > v1) {
            // Not a partition of the verbs: the caller strokes the batch path by path.
            if (lane == 0) S.words[1] = S.words[STROKE_VERBS_UNFIT] = 1u;
        } else if (ve - vb > 64u) {
            prepare_path<8>(A, S, path, v0, vb, ve, lane);
        } else {
            prepare_path<1>(A, S, path, v0, vb, ve, lane);
        }
    }
}

// ---- 2. sharp turns ----------------------------------------------------------------------------
// Whether find_sharp_turn (geom.cuh) gets past its first tests, which decide most quadratics.
__device__ __forceinline__ bool may_turn(V2 from, V2 ctrl, V2 to) {
    const V2 baseline = to - from, v = ctrl - from;
    const V2 n = V2{-baseline.y, baseline.x};
    const float vb = dot(v, baseline), vn = dot(v, n);
    if ((vb >= 0.0f && vb <= dot(baseline, baseline)) || fabsf(vn) * 2.0f >= fabsf(vb))
        return !(sqlen(baseline) * 30.0f > sqlen(v));
    return true;
}

constexpr uint32_t TURN_TILE = 2048;
__global__ void __launch_bounds__(256) turns_kernel(StrokeArgs A, StrokeVerbs S) {
    __shared__ uint32_t list[TURN_TILE];
    __shared__ uint32_t count;
    const uint32_t nv = batch_verbs(A);
    if (unfit(S, nv)) return;
    for (uint32_t tile = blockIdx.x * TURN_TILE; tile < nv; tile += gridDim.x * TURN_TILE) {
        __syncthreads();
        if (threadIdx.x == 0) count = 0;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < TURN_TILE; i += blockDim.x) {
            const uint32_t v = tile + i;
            if (v >= nv || (S.kind[v] & KIND_MASK) != LYON_VERB_QUADRATIC_TO) continue;
            const uint32_t p = S.rec[v];
            if (may_turn(load_pt(A.points, p - 1), load_pt(A.points, p), load_pt(A.points, p + 1)))
                list[atomicAdd(&count, 1u)] = v;
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) {
            const uint32_t v = list[i], p = S.rec[v];
            float ts;
            if (find_sharp_turn(load_pt(A.points, p - 1), load_pt(A.points, p),
                                load_pt(A.points, p + 1), &ts)) {
                S.flags[v] = (uint16_t)VF_TURN;
                S.cut[v] = __float_as_uint(ts);
            }
        }
    }
}

// ---- 3. walk -----------------------------------------------------------------------------------

// The merge chain of an irregular verb after the kept point `c1` (stroke.rs:1530-1536).
struct Chain {
    V2 first1, first2, last, before, before2;
    uint32_t kept;
    bool flat1, lastflat, beforeflat, end_kept;
    // A verb that can be cut all the same: one row of steps merges into one interior point, or
    // one interior join is no flattening step, and nothing else is out of the ordinary.
    bool cuttable;
    uint32_t at, gap;  // the point and the steps merged into it
};
__device__ __noinline__ void replay_chain(Unit a, const Unit& b, V2 c1, float thr, float hw,
                                          Chain& c) {
    c.first1 = c.first2 = c.last = c.before = c.before2 = c1;
    c.kept = 0;
    c.flat1 = c.lastflat = c.beforeflat = c.end_kept = false;
    c.cuttable = b.m == 0;
    c.at = c.gap = 0;
    uint32_t last_k = 0;
    const uint32_t units = b.m > 0 ? 2u : 1u;
    for (uint32_t u = 0; u < units; ++u) {
        float t = a.t0;
        for (uint32_t k = 1; k <= a.m; ++k) {
            V2 q = a.to;
            bool flat = false;
            if (k < a.m) {
                t = t + a.s;
                q = poly_sample(a.p, t);
                flat = t != 1.0f;
                c.cuttable &= flat;
            }
            c.end_kept = !too_close(c.last, q, thr);
            if (!c.end_kept) {
                c.cuttable &= last_k > 0 && (c.at == 0 || c.at == last_k);
                c.at = last_k;
                ++c.gap;
                continue;
            }
            if (c.kept > 0) {
                const V2 pe = c.last - c.before, e = q - c.last;
                if (!(dot(pe, e) > 0.0f)) {
                    c.cuttable &= c.at == 0 || c.at == last_k;
                    c.at = last_k;
                } else {
                    c.cuttable &= skip_impossible(c.before, c.last, pe, hw);
                }
            }
            if (c.kept == 0) {
                c.first1 = q;
                c.flat1 = flat;
            } else if (c.kept == 1) {
                c.first2 = q;
            }
            c.before2 = c.before;
            c.before = c.last;
            c.beforeflat = c.lastflat;
            c.last = q;
            c.lastflat = flat;
            last_k = k;
            ++c.kept;
        }
        a = b;
    }
    c.cuttable &= c.end_kept && c.at > 0 && c.at <= 0xFFFFu && c.gap <= 0xFFFFu;
}
__device__ __forceinline__ void store_chain(const StrokeVerbs& S, uint32_t v, uint32_t path,
                                            uint32_t keep_flags, const Chain& c) {
    S.firsts[v] = make_float4(c.first1.x, c.first1.y, c.first2.x, c.first2.y);
    S.lasts[v] = make_float4(c.before.x, c.before.y, c.before2.x, c.before2.y);
    uint32_t f = keep_flags | (c.flat1 ? VF_FLAT1 : 0u) | (c.beforeflat ? VF_FLATL : 0u) |
                 (min(c.kept, 3u) << VF_NK_SHIFT);
    if (c.kept == 0) leave_to_walk(S, path);
    if (!c.end_kept) {
        f |= VF_MERGED | (c.lastflat ? VF_ENDFLAT : 0u);
        S.fin[v] = make_float2(c.last.x, c.last.y);
    }
    S.flags[v] = (uint16_t)f;
}

// The most steps of an irregular verb: beyond, its path is left to the walk, which takes 32 steps at a
// time. For count and emit pass together a thread takes 1 to 2.6 us a step, the walk 0.13 us a step,
// 3.4 us a verb of the path and, once a batch, 100 us of further launches; in a large batch the other
// verbs take longer than that one thread. The replay that finds whether the verb can be cut instead
// takes 0.3 us a step: it is tried for REPLAY_STEPS times as many where points merge at one cusp or
// none (a drawn cusp; what else there is can hardly be cut). One path of one curve that turns round
// twice, 1,864 steps: 1266 -> 434 us, by the walk 338; 2,000 paths of ten such curves of 590 steps 3527
// -> 1200 us, by the walk 976.
__device__ __forceinline__ uint32_t serial_steps(const StrokeArgs& A, uint32_t path, uint32_t nv) {
    const uint32_t verbs = A.verb_offsets[path + 1] - A.verb_offsets[path];
    return max(64u + verbs + verbs / 2u, nv / 500u);
}
constexpr uint32_t REPLAY_STEPS = 8;

struct WalkSlot {
    UnitSmem u;
    float thr, hw;
    uint32_t store;  // the verb's slot when it is this one unit: its points next to the ends go
                     // straight out; else NO_STORE
    uint32_t rough;  // some point merges
    uint32_t skip;   // some skip is not ruled out
    uint32_t bad, badk;  // interior joins that are no flattening steps, one of them
    uint32_t pad;
};
constexpr uint32_t NO_STORE = 0xFFFFFFFFu;
struct WalkSmem {
    WalkSlot unit[WIN_UNITS];
    PointSmem pt;
};

// Bound by instruction issue: about a hundred per 32 points, and the set-up of the windows.
__global__ void __launch_bounds__(WIN_WARPS * 32) walk_kernel(StrokeArgs A, StrokeVerbs S) {
    extern __shared__ __align__(16) unsigned char walk_smem[];
    const int lane = threadIdx.x & 31;
    WalkSmem& sm = reinterpret_cast<WalkSmem*>(walk_smem)[threadIdx.x >> 5];
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t nv = batch_verbs(A);
    if (unfit(S, nv)) return;
    const uint32_t W = window_verbs(nv, nwarps);
    for (uint32_t w0 = warp * W; w0 < nv; w0 += nwarps * W) {
        const uint32_t v = w0 + (uint32_t)lane;
        Unit a, b;
        a.m = b.m = 0;
        uint32_t path = 0, flags = 0;
        V2 c1 = V2{0.0f, 0.0f};
        float thr = 0.0f, hw = 0.0f;
        if ((uint32_t)lane < W && v < nv) {
            const int kind = S.kind[v] & KIND_MASK;
            if (is_segment(kind)) {
                path = S.path[v];
                c1 = end_point(S, A.points, v - 1);
                if (kind == LYON_VERB_LINE_TO) {
                    const V2 E = load_pt(A.points, S.rec[v]);
                    S.firsts[v] = make_float4(E.x, E.y, 0.0f, 0.0f);
                    S.lasts[v] = make_float4(c1.x, c1.y, 0.0f, 0.0f);
                    S.flags[v] = (uint16_t)(1u << VF_NK_SHIFT);
                    S.vpre[v] = 0;
                    S.ipre[v] = 0;
                } else {
                    const StrokeParams P = make_params(A.options[A.num_options > 1 ? path : 0]);
                    thr = P.merge_threshold;
                    hw = P.hw;
                    flags = S.flags[v];
                    verb_units(kind, S.rec[v], A.points, P.tolerance, flags,
                               flags & VF_TURN ? S.cut[v] : 0u, a, b);
                    if (a.m > MAX_SERIAL_STEPS || b.m > MAX_SERIAL_STEPS) {
                        leave_to_walk(S, path);
                        a.m = b.m = 0;
                    }
                }
            }
        }
        const bool ra = a.m > 0, rb = b.m > 0;
        const uint32_t mask_a = __ballot_sync(FULL, ra), mask_b = __ballot_sync(FULL, rb);
        if (mask_a == 0) continue;
        const uint32_t below = (1u << lane) - 1u;
        const uint32_t slot = __popc(mask_a & below) + __popc(mask_b & below);
        const uint32_t nunits = __popc(mask_a) + __popc(mask_b);
        const uint32_t steps = a.m + b.m;
        uint32_t incl = steps;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t up = __shfl_up_sync(FULL, incl, d);
            if (lane >= d) incl += up;
        }
        const uint32_t total = __shfl_sync(FULL, incl, 31);
        const uint32_t excl = incl - steps;
        for (uint32_t i = 0; i < (ra ? rb ? 2u : 1u : 0u); ++i) {
            WalkSlot& r = sm.unit[slot + i];
            lay_out_unit(r.u, i ? b : a, i ? a.to : c1, excl + (i ? a.m : 0u));
            r.thr = thr;
            r.hw = hw;
            r.store = rb ? NO_STORE : v;
            r.rough = r.skip = r.bad = r.badk = 0;
        }
        __syncwarp();
        V2 q = V2{0.0f, 0.0f}, ne = V2{0.0f, 0.0f};
        for (uint32_t r0 = 0; r0 < total; r0 += WIN_ROUND) {
            const uint32_t rn = min(WIN_ROUND, total - r0);
            fill_points(sm.pt, &sm.unit[0].u, sizeof(WalkSlot), nunits, r0, rn, lane);
            for (uint32_t cb = 0; cb < rn; cb += 32) {
                const uint32_t at = cb + (uint32_t)lane;
                const uint32_t i = min(at, rn - 1u);
                WalkSlot& r = sm.unit[sm.pt.owner[i]];
                const uint32_t k = r0 + i - r.u.excl + 1u, m = r.u.m_cubic >> 1;
                const float t = sm.pt.t[i];
                const V2 old_q = q, old_e = ne;
                q = unit_point(r.u, k, t);
                V2 qp = V2{from_left(q.x, old_q.x, lane), from_left(q.y, old_q.y, lane)};
                if (k == 1u) {
                    const float4 e = r.u.c1_to;
                    qp = V2{e.x, e.y};
                }
                ne = q - qp;
                const V2 pe = V2{from_left(ne.x, old_e.x, lane), from_left(ne.y, old_e.y, lane)};
                if (at < rn) {
                    // The join at this point, when it is interior: whether lyon steps it as a
                    // flattened point (a parameter of exactly 1 is an end), and its skip test.
                    if (sqlen(ne) < r.thr || (k < m && t == 1.0f)) r.rough = 1u;
                    if (k < m && !skip_impossible(qp, q, ne, r.hw)) r.skip = 1u;
                    // The join at the point before.
                    if (k > 1u && !(dot(pe, ne) > 0.0f)) {
                        atomicAdd(&r.bad, 1u);
                        r.badk = k - 1u;
                    }
                    if ((k <= 2u || k + 1u >= m) && r.store != NO_STORE) {
                        float2* f = reinterpret_cast<float2*>(S.firsts + r.store);
                        float2* l = reinterpret_cast<float2*>(S.lasts + r.store);
                        if (k <= 2u) f[k - 1u] = make_float2(q.x, q.y);
                        if (k + 1u >= m) l[m - k] = make_float2(qp.x, qp.y);
                    }
                }
            }
            __syncwarp();
        }
        if (ra) {
            const WalkSlot& x = sm.unit[slot];
            uint32_t rough = x.rough, skip = x.skip, bad = x.bad, badk = x.badk;
            if (rb) {
                rough |= sm.unit[slot + 1].rough;
                skip |= sm.unit[slot + 1].skip;
                bad += sm.unit[slot + 1].bad;
            }
            // One cusp cuts the verb in two runs, unless it is split already. (A clipped miter there
            // leaves sides that are not symmetric, as the skip test's bound wants them:
            // extra_count_kernel evaluates the test at the join after it.)
            const bool irregular = rough || skip || bad > 1 || (bad == 1 && rb);
            // (The walk of a variable-width path is one thread's as well.)
            const uint32_t most = irregular && !A.widths ? serial_steps(A, path, nv) : steps;
            const bool refused = skip && !rough && bad == 0 && !rb;  // walk_irregular comes to that
            if ((refused && !A.widths) || steps > (rough && bad <= 1 && !rb ? REPLAY_STEPS * most : most)) {
                leave_to_walk(S, path);
            } else if (irregular) {
                Chain c;
                replay_chain(a, b, c1, thr, hw, c);
                if (c.cuttable) {
                    store_chain(S, v, path, VF_CUT | (c.at + c.gap + 1u == a.m ? VF_SECOND1 : 0u),
                                c);
                    S.cut[v] = c.at | (c.gap << 16);
                    S.extra[atomicAdd(&S.words[6], 1u)] = v;
                    if (a.m > c.gap + 2u) S.words[3] = 1u;
                } else if (steps > most) {
                    leave_to_walk(S, path);
                } else {
                    store_chain(S, v, path, VF_IRR | (flags & VF_TURN), c);
                    if (!c.end_kept) S.drops[atomicAdd(&S.words[4], 1u)] = v;
                    S.irregular[atomicAdd(&S.words[7], 1u)] = v;
                }
            } else {
                uint32_t f = (flags & VF_TURN) | (min(steps, 3u) << VF_NK_SHIFT);
                if (a.m >= 2) f |= VF_FLAT1;
                if ((rb ? b.m : a.m) >= 2) f |= VF_FLATL;
                if (bad == 1) {
                    f |= VF_CUT;
                    S.cut[v] = badk;
                    if (badk + 1u == a.m) f |= VF_SECOND1;
                }
                if (rb) {
                    if (b.m == 1) f |= VF_SECOND1;
                    const V2 f1 = first_point(a), l1 = point_before_end(b, a.to);
                    const V2 f2 = a.m >= 3 ? poly_sample(a.p, (0.0f + a.s) + a.s)
                                           : a.m == 2 ? a.to : first_point(b);
                    const V2 l2 = b.m >= 3 ? poly_sample(b.p, unit_t(b, b.m - 2))
                                           : b.m == 2 ? a.to : point_before_end(a, c1);
                    S.firsts[v] = make_float4(f1.x, f1.y, f2.x, f2.y);
                    S.lasts[v] = make_float4(l1.x, l1.y, l2.x, l2.y);
                }
                S.flags[v] = (uint16_t)f;
                if (f & VF_TWO) {
                    S.extra[atomicAdd(&S.words[6], 1u)] = v;
                } else {
                    // The interior joins' vertices and triangles.
                    S.vpre[v] = 2u * (a.m - 1u);
                    S.ipre[v] = a.m >= 2 ? 2u * (a.m - 2u) : 0u;
                }
                if (steps > (rb ? 2u : 1u)) S.words[3] = 1u;
            }
        }
        __syncwarp();
    }
}

// A verb whose end point merged leaves the next verb another point to start from than
// walk_kernel took: its chain again from there.
__global__ void __launch_bounds__(128) drops_kernel(StrokeArgs A, StrokeVerbs S) {
    if (unfit(S, batch_verbs(A))) return;
    const uint32_t n = S.words[4];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t v = S.drops[i], next = v + 1, path = S.path[v];
        const int kind = S.kind[next] & KIND_MASK;
        // Lines dropped after it were compared with the end point that merged.
        if (S.kind[next] & KIND_GAP) leave_to_walk(S, path);
        if (S.path_walk[path] || !is_segment(kind)) continue;
        const uint32_t flags = S.flags[next];
        const float2 f = S.fin[v];
        const V2 c1 = V2{f.x, f.y};
        const StrokeParams P = make_params(A.options[A.num_options > 1 ? path : 0]);
        if (flags & VF_MERGED) {
            leave_to_walk(S, path);  // two in a row
        } else if (kind == LYON_VERB_LINE_TO) {
            if (too_close(c1, load_pt(A.points, S.rec[next]), P.merge_threshold))
                leave_to_walk(S, path);
            S.lasts[next] = make_float4(c1.x, c1.y, 0.0f, 0.0f);
        } else {
            Unit a, b;
            verb_units(kind, S.rec[next], A.points, P.tolerance, flags & VF_TURN, S.cut[next], a, b);
            Chain c;
            replay_chain(a, b, c1, P.merge_threshold, P.hw, c);
            if (!c.end_kept) leave_to_walk(S, path);
            store_chain(S, next, path, VF_IRR | (flags & VF_TURN), c);
            // (In the other list, if it is there, it counts for nothing now.)
            if (!(flags & VF_IRR)) S.irregular[atomicAdd(&S.words[7], 1u)] = next;
        }
    }
}

// ---- joins -------------------------------------------------------------------------------------

// Adds up a verb's joins in order: vertices, triangles (without the edge into the verb's first
// join, which the prefix pass or the emit pass knows from the verb before), and the id structures
// at both ends.
struct JoinSum {
    uint32_t v, tris, to_first, from_f;
    bool have;
    __device__ __forceinline__ void init() {
        v = tris = to_first = from_f = 0;
        have = false;
    }
    __device__ __forceinline__ void add(uint32_t vertices, uint32_t join_tris, uint32_t to_f,
                                        uint32_t from) {
        if (have) {
            tris += edge_count_flags(from_f, to_f);
        } else {
            to_first = to_f;
            have = true;
        }
        v += vertices;
        tris += join_tris;
        from_f = from;
    }
    __device__ __forceinline__ void run(uint32_t joins) {  // flattening-step joins in a row
        if (joins == 0) return;
        add(2, 0, 0, 0);
        v += 2 * (joins - 1);
        tris += 2 * (joins - 1);
    }
};

// Where a verb's output goes (emit phase) and the ids its next edge starts from.
struct VerbOut {
    PathOut po;
    uint32_t vo, io;      // next vertex and index of the path
    uint32_t pfn, pfp;
    bool edge;            // the next join has an edge into it
    int st;
    float adv;            // the advancement of the next join (records only)
};

// REC: attribute records instead of positions (here and in the kernels of the emit phase).
template <bool REC>
__device__ __forceinline__ SinkT<REC> sink_at(const PathOut& po, uint32_t vo, uint32_t io) {
    SinkT<REC> s;
    s.id_base = po.id_base + vo;
    s.nv = 0;
    s.ni = 0;
    s.vout = REC ? nullptr : po.vout + vo;
    s.rout = REC ? po.rout + vo : nullptr;
    s.iout = po.bits == 16 ? (void*)((uint16_t*)po.iout + io) : (void*)((uint32_t*)po.iout + io);
    s.index_bits = po.bits;
    s.vcap = cap_left(po.vmax, vo);
    s.icap = cap_left(po.imax, io);
    s.overflow = false;
    return s;
}

template <bool REC>
__device__ __forceinline__ void emit_general(VerbOut& o, V2 prv, V2 cur, bool flat, V2 nxt,
                                             const StrokeParams& P, uint32_t packed) {
    SinkT<REC> sk = sink_at<REC>(o.po, o.vo, o.io);
    if (REC) sk.adv = o.adv;
    const JoinEmitOut r = slow_join_emit_at(prv, cur, flat, nxt, P, sk, o.edge, o.pfn, o.pfp);
    if (r.st != LYON_OK) o.st = r.st;
    if (r.overflow || r.nv != pj_vertices(packed)) o.st = LYON_ERR_INTERNAL;
    const uint32_t base = o.po.id_base + o.vo;
    o.pfn = base + pj_neg(packed);
    o.pfp = base + pj_pos(packed);
    o.vo += r.nv;
    o.io += r.ni;
    o.edge = true;
}

// A flattening step's join (stroke.rs:1743-1806) written through `o`.
template <bool REC>
__device__ __forceinline__ void emit_step(VerbOut& o, V2 prv, V2 cur, V2 nxt, float hw) {
    const SidePair s = fast_join_sides(prv, cur, nxt, hw);
    SinkT<REC> sk = sink_at<REC>(o.po, o.vo, o.io);
    V2 n = V2{0.0f, 0.0f};
    if (REC) {  // (the positions are at n and -n times the half width)
        const V2 pe = cur - prv, ne = nxt - cur;
        n = compute_normal(pe / vlength(pe), ne / vlength(ne));
        sk.adv = o.adv;
    }
    const uint32_t id = sk.vertex(s.pn, n, SP);
    sk.vertex(s.nn, -n, SN);
    if (o.edge) edge_triangles(o.pfn, o.pfp, id + 1, id, &sk);
    if (sk.overflow) o.st = LYON_ERR_INTERNAL;
    o.vo += sk.nv;
    o.io += sk.ni;
    o.pfn = id + 1;
    o.pfp = id;
    o.edge = true;
}

// The walk of one irregular verb by one thread: lyon's step over its flattened points from the
// kept point `c1` before it (the join at c1 belongs to the verb before, the one at the last kept
// point is not done here). Counts into `sum`, or emits through `o`. Returns false, counting, when the
// path has to be walked as a whole: a join fails, or the skip test fires or is not ruled out by its
// bound. (After a clipped miter, whose sides are not symmetric, the test is evaluated; at the first
// join by the verb before, first_step_skips.)
template <bool EMIT, bool REC>
__device__ __noinline__ bool walk_irregular(Unit a, const Unit& b, V2 c1, const StrokeParams& P,
                                            JoinSum& sum, VerbOut* o, uint32_t* last_join) {
    V2 cur = c1, prv = c1, jpn = c1, jnn = c1;
    bool curflat = false, sym = true;  // of the join at prv, with the sides (jpn, jnn) if not
    uint32_t kept = 0;
    const uint32_t units = b.m > 0 ? 2u : 1u;
    for (uint32_t u = 0; u < units; ++u) {
        float t = a.t0;
        for (uint32_t k = 1; k <= a.m; ++k) {
            V2 q = a.to;
            bool flat = false;
            if (k < a.m) {
                t = t + a.s;
                q = poly_sample(a.p, t);
                flat = t != 1.0f;
            }
            if (too_close(cur, q, P.merge_threshold)) continue;
            if (kept > 0) {
                const V2 pe = cur - prv, ne = q - cur;
                if (curflat && dot(pe, ne) > 0.0f) {
                    if (!EMIT && (sym ? !skip_impossible(prv, cur, pe, P.hw)
                                      : skip_fires(prv, jpn, jnn, cur, q, P.hw)))
                        return false;
                    if (EMIT) {
                        emit_step<REC>(*o, prv, cur, q, P.hw);
                    } else {
                        sum.add(2, 0, 0, 0);
                        *last_join = PACKED_STEP;
                    }
                    sym = true;
                } else {
                    const SlowJoin sj = slow_join_summary(prv, cur, curflat, q, P);
                    uint32_t packed;
                    if (!pack_join(sj, &packed)) return false;
                    jpn = sj.pn;
                    jnn = sj.nn;
                    if (EMIT) {
                        emit_general<REC>(*o, prv, cur, curflat, q, P, packed);
                    } else {
                        sum.add(sj.vcount, sj.jtris, sj.to_f, sj.from_f);
                        *last_join = packed;
                    }
                    sym = sj.sym;
                }
            }
            if (EMIT && REC) o->adv = o->adv + vlength(q - cur);
            prv = cur;
            cur = q;
            curflat = flat;
            ++kept;
        }
        a = b;
    }
    return true;
}

// The next segment's first flattening-step join comes right after the general join at `cur`: with
// a clipped miter there its side points are not symmetric, and the skip test is evaluated.
__device__ __forceinline__ bool first_step_skips(const StrokeVerbs& S, uint32_t next, V2 cur,
                                                 const SlowJoin& sj, float hw) {
    const uint32_t f = S.flags[next];
    if (sj.sym || !(f & VF_FLAT1) || flags_nk(f) < 2) return false;
    const float4 q = S.firsts[next];
    const V2 q1 = V2{q.x, q.y}, q2 = V2{q.z, q.w};
    if (!(dot(q1 - cur, q2 - q1) > 0.0f)) return false;
    return skip_fires(cur, sj.pn, sj.nn, q1, q2, hw);
}

// Whether the join at a verb's last kept point is a flattening step (its end point merged).
__device__ __forceinline__ bool end_steps(uint32_t flags, V2 last, V2 cur, V2 nxt) {
    return (flags & VF_ENDFLAT) && dot(cur - last, nxt - cur) > 0.0f;
}

// 4. The verbs with something but a run inside (`extra`: cusps, sharp turns, irregular verbs; a
// twelfth of a drawing's, gathered so that full warps do them): their interior sums in vpre and
// ipre (triangles), and in `split` the join between the two runs, or an irregular verb's last
// interior join.
__global__ void __launch_bounds__(128) extra_count_kernel(StrokeArgs A, StrokeVerbs S) {
    if (unfit(S, batch_verbs(A))) return;
    // The verbs of two runs, then, from a warp's boundary, the irregular ones.
    const uint32_t n2 = S.words[6], start = (n2 + 31u) & ~31u, n = start + S.words[7];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (i >= n2 && i < start) continue;
        const uint32_t v = i < n2 ? S.extra[i] : S.irregular[i - start];
        const uint32_t path = S.path[v], flags = S.flags[v];
        if ((i < n2) == ((flags & VF_IRR) != 0)) continue;
        if (S.path_walk[path]) continue;
        const StrokeParams P = make_params(A.options[A.num_options > 1 ? path : 0]);
        JoinSum sum;
        sum.init();
        bool ok = true;
        Unit a, b;
        verb_units(S.kind[v] & KIND_MASK, S.rec[v], A.points, P.tolerance, flags,
                   flags & VF_TWO ? S.cut[v] : 0u, a, b);
        const V2 c1 = last_kept(S, A.points, v - 1);
        uint32_t packed = PACKED_STEP;
        if (flags & VF_IRR) {
            ok = walk_irregular<false, false>(a, b, c1, P, sum, nullptr, &packed);
        } else {
            sum.run(a.m - 1);
            const V2 before = point_before_end(a, c1), after = first_point(b);
            if ((flags & VF_CUT) && dot(a.to - before, after - a.to) > 0.0f) {
                sum.run(1);  // steps merged here, and the join is still a flattening step
            } else {
                const SlowJoin sj = slow_join_summary(before, a.to, (flags & VF_CUT) != 0, after, P);
                ok = pack_join(sj, &packed);
                if (!sj.sym && b.m >= 2) {
                    const V2 q2 = b.m >= 3 ? poly_sample(b.p, (b.t0 + b.s) + b.s) : b.to;
                    if (skip_fires(a.to, sj.pn, sj.nn, after, q2, P.hw)) ok = false;
                }
                sum.add(sj.vcount, sj.jtris, sj.to_f, sj.from_f);
            }
            sum.run(b.m - 1);
        }
        S.split[v] = packed;
        if (!ok) leave_to_walk(S, path);
        if (sum.to_first) S.flags[v] = (uint16_t)(flags | VF_TOFIRST);
        S.vpre[v] = sum.v;
        S.ipre[v] = sum.tris;
    }
}

// The last interior join of a verb that has one (NK >= 2), packed.
__device__ __forceinline__ uint32_t last_interior(const StrokeVerbs& S, uint32_t v,
                                                  uint32_t flags) {
    return (flags & VF_IRR) || ((flags & VF_TWO) && (flags & VF_SECOND1)) ? S.split[v]
                                                                          : PACKED_STEP;
}

// 5. The join at each verb's end, one verb per thread. Bound by the general join's arithmetic
// (about a thousand instructions with a round join), which every lane of a warp runs at once.
__global__ void __launch_bounds__(256) joins_count_kernel(StrokeArgs A, StrokeVerbs S) {
    const uint32_t nv = batch_verbs(A);
    if (unfit(S, nv)) return;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nv;
         v += gridDim.x * blockDim.x) {
        if (!is_segment(S.kind[v] & KIND_MASK)) continue;
        const uint32_t path = S.path[v];
        if (S.path_walk[path]) continue;
        uint32_t tris = S.ipre[v];
        if (is_segment(S.kind[v + 1] & KIND_MASK)) {
            const uint32_t flags = S.flags[v];
            const StrokeParams P = make_params(A.options[A.num_options > 1 ? path : 0]);
            const float4 f = S.firsts[v + 1], l = S.lasts[v];
            const V2 nxt = V2{f.x, f.y}, last = V2{l.x, l.y}, cur = last_kept(S, A.points, v);
            uint32_t packed = PACKED_STEP;
            bool ok = true;
            if (end_steps(flags, last, cur, nxt)) {
                ok = P.line_join != LYON_JOIN_MITER_CLIP &&
                     skip_impossible(last, cur, cur - last, P.hw);
            } else {
                const SlowJoin sj = slow_join_summary(last, cur, (flags & VF_ENDFLAT) != 0, nxt, P);
                ok = pack_join(sj, &packed) && !first_step_skips(S, v + 1, cur, sj, P.hw);
            }
            if (!ok) leave_to_walk(S, path);
            S.join[v] = packed;
            S.vpre[v] += pj_vertices(packed);
            tris += pj_tris(packed);
            if (flags_nk(flags) >= 2) {
                tris += edge_count_flags(pj_from(last_interior(S, v, flags)), pj_to(packed));
            } else if (pj_to(packed)) {
                // Its only join is its first one. Readers of the flags look at other bits.
                S.flags[v] = (uint16_t)(flags | VF_TOFIRST);
            }
        }
        S.ipre[v] = 3u * tris;
    }
}

// The position of a verb's output and the edge into its first join.
template <bool REC>
__device__ __forceinline__ void verb_out(const StrokeArgs& A, const StrokeVerbs& S, uint32_t v,
                                         uint32_t path, VerbOut& o) {
    o.po = path_out<true, REC>(A, path);
    o.adv = REC ? S.adv[v - 1].w : 0.0f;
    o.vo = S.vpre[v] - S.path_v[path];
    o.io = S.ipre[v] - S.path_i[path];
    o.st = LYON_OK;
    o.edge = (S.kind[v - 1] & KIND_MASK) != LYON_VERB_BEGIN;
    o.pfn = o.pfp = INVALID_ID;
    if (o.edge) {
        const uint32_t j = S.join[v - 1];
        const uint32_t base = o.po.id_base + o.vo - pj_vertices(j);
        o.pfn = base + pj_neg(j);
        o.pfp = base + pj_pos(j);
    }
}

// Triangles of the edge into a flattening-step join after ids (pfn, pfp).
__device__ __forceinline__ uint32_t edge_into_step(const VerbOut& o) {
    return o.edge ? edge_count_flags(o.pfn == o.pfp ? EF_SELF_EQ : 0u, 0u) : 0u;
}

// Steps over the output of a run of flattening-step joins (written by runs_kernel).
__device__ __forceinline__ void pass_run(VerbOut& o, uint32_t joins) {
    if (joins == 0) return;
    o.io += 3u * (edge_into_step(o) + 2u * (joins - 1u));
    o.vo += 2u * joins;
    o.pfn = o.po.id_base + o.vo - 1u;
    o.pfp = o.pfn - 1u;
    o.edge = true;
}

// Output of the verbs in `extra` but for their runs.
template <bool REC>
__global__ void __launch_bounds__(128) extra_emit_kernel(StrokeArgs A, StrokeVerbs S) {
    if (batch_verbs(A) > S.cap) return;
    // The verbs of two runs, then, from a warp's boundary, the irregular ones.
    const uint32_t n2 = S.words[6], start = (n2 + 31u) & ~31u, n = start + S.words[7];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (i >= n2 && i < start) continue;
        const uint32_t v = i < n2 ? S.extra[i] : S.irregular[i - start];
        const uint32_t path = S.path[v], flags = S.flags[v];
        if ((i < n2) == ((flags & VF_IRR) != 0)) continue;
        if (S.path_walk[path] || A.status[path] != LYON_OK) continue;
        const StrokeParams P = make_params(A.options[A.num_options > 1 ? path : 0]);
        VerbOut o;
        verb_out<REC>(A, S, v, path, o);
        Unit a, b;
        verb_units(S.kind[v] & KIND_MASK, S.rec[v], A.points, P.tolerance, flags,
                   flags & VF_TWO ? S.cut[v] : 0u, a, b);
        const V2 c1 = last_kept(S, A.points, v - 1);
        if (flags & VF_IRR) {
            JoinSum none;
            none.init();
            uint32_t last;
            if (!walk_irregular<true, REC>(a, b, c1, P, none, &o, &last))
                o.st = LYON_ERR_INTERNAL;
        } else {
            pass_run(o, a.m - 1);
            if (REC) o.adv = S.adv[v].x;
            const V2 before = point_before_end(a, c1), after = first_point(b);
            if ((flags & VF_CUT) && dot(a.to - before, after - a.to) > 0.0f) {
                emit_step<REC>(o, before, a.to, after, P.hw);
            } else {
                emit_general<REC>(o, before, a.to, (flags & VF_CUT) != 0, after, P, S.split[v]);
            }
        }
        if (o.st != LYON_OK) A.status[path] = o.st;
    }
}

// Output of the join at each verb's end, one verb per thread. It is the last thing of the verb.
template <bool REC>
__global__ void __launch_bounds__(256) joins_emit_kernel(StrokeArgs A, StrokeVerbs S) {
    const uint32_t nv = batch_verbs(A);
    if (nv > S.cap) return;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nv;
         v += gridDim.x * blockDim.x) {
        if (!is_segment(S.kind[v] & KIND_MASK) || !is_segment(S.kind[v + 1] & KIND_MASK)) continue;
        const uint32_t path = S.path[v];
        if (S.path_walk[path] || A.status[path] != LYON_OK) continue;
        const uint32_t flags = S.flags[v], join = S.join[v];
        const StrokeParams P = make_params(A.options[A.num_options > 1 ? path : 0]);
        VerbOut o;
        o.po = path_out<true, REC>(A, path);
        o.st = LYON_OK;
        o.adv = REC ? S.adv[v].w : 0.0f;
        o.edge = true;
        uint32_t prev = PACKED_STEP;
        if (flags_nk(flags) >= 2) {
            prev = last_interior(S, v, flags);
        } else if ((S.kind[v - 1] & KIND_MASK) == LYON_VERB_BEGIN) {
            o.edge = false;
        } else {
            prev = S.join[v - 1];
        }
        const uint32_t edge = o.edge ? edge_count_flags(pj_from(prev), pj_to(join)) : 0u;
        const uint32_t end_v = S.vpre[v + 1] - S.path_v[path];
        const uint32_t end_i = S.ipre[v + 1] - S.path_i[path];
        o.vo = end_v - pj_vertices(join);
        o.io = end_i - 3u * (edge + pj_tris(join));
        const uint32_t base = o.po.id_base + o.vo - pj_vertices(prev);
        o.pfn = base + pj_neg(prev);
        o.pfp = base + pj_pos(prev);
        const float4 f = S.firsts[v + 1], l = S.lasts[v];
        const V2 nxt = V2{f.x, f.y}, last = V2{l.x, l.y}, cur = last_kept(S, A.points, v);
        if (end_steps(flags, last, cur, nxt)) {
            emit_step<REC>(o, last, cur, nxt, P.hw);
        } else {
            emit_general<REC>(o, last, cur, (flags & VF_ENDFLAT) != 0, nxt, P, join);
        }
        if (o.st != LYON_OK || o.vo != end_v || o.io != end_i)
            A.status[path] = o.st != LYON_OK ? o.st : LYON_ERR_INTERNAL;
    }
}

// ---- 5. tails ----------------------------------------------------------------------------------

// The TailJob of the sub-path that ends in slot v, from the recorded points.
template <bool REC>
__device__ __forceinline__ TailJob tail_job(const StrokeArgs& A, const StrokeVerbs& S, uint32_t v,
                                            uint32_t path, const StrokeParams& P, bool emit) {
    const uint32_t kind = S.kind[v];
    const uint32_t b = S.rec[v];  // the Begin's slot
    TailJob j;
    j.path = path;
    j.flags = ((kind & KIND_MASK) == LYON_VERB_CLOSE ? TJ_CLOSED : 0u) |
              (kind & KIND_MNEC ? TJ_MNEC : 0u);
    j.adv0 = j.adv1 = j.adv2 = REC ? S.adv[b].w : 0.0f;
    j.vcur = emit ? S.vpre[v] - S.path_v[path] : 0u;
    j.icur = emit ? S.ipre[v] - S.path_i[path] : 0u;
    j.base1 = j.jbase = 0;
    j.p0 = end_point(S, A.points, b);
    j.p1 = j.p2 = j.c1 = j.c2 = j.c3 = j.p0;
    j.n = 1;
    const uint32_t segs = v - b - 1;
    if (segs == 0) return j;
    const uint32_t f1 = S.flags[b + 1], fl = S.flags[v - 1];
    j.n += flags_nk(f1) + (segs > 1 ? flags_nk(S.flags[b + 2]) : 0u) + (segs > 2 ? 1u : 0u);
    j.c1 = last_kept(S, A.points, v - 1);
    if (REC) {
        const float4 a = S.adv[v - 1];
        j.adv1 = a.w;
        j.adv2 = flags_nk(fl) >= 2 ? a.z : S.adv[v - 2].w;
    }
    if (fl & VF_ENDFLAT) j.flags |= TJ_F1;
    const float4 fs = S.firsts[b + 1], ls = S.lasts[v - 1];
    j.p1 = V2{fs.x, fs.y};
    j.c2 = V2{ls.x, ls.y};
    if (j.n == 2) return j;
    const bool flat1 = (f1 & VF_FLAT1) != 0;
    if (flags_nk(f1) >= 2) {
        j.p2 = V2{fs.z, fs.w};
    } else {
        const float4 g = S.firsts[b + 2];
        j.p2 = V2{g.x, g.y};
    }
    bool flat2 = false;
    if (flags_nk(fl) >= 2) {
        j.c3 = V2{ls.z, ls.w};
        flat2 = (fl & VF_FLATL) != 0;
    } else {
        // One kept point: the one before it is the last of the verb before.
        const float4 g = S.lasts[v - 2];
        j.c3 = V2{g.x, g.y};
        flat2 = (S.flags[v - 2] & VF_ENDFLAT) != 0;
    }
    const bool fast1 = flat1 && dot(j.p1 - j.p0, j.p2 - j.p1) > 0.0f;
    const bool fast2 = flat2 && dot(j.c2 - j.c3, j.c1 - j.c2) > 0.0f;
    j.flags |= (flat1 ? TJ_FLAT1 : 0u) | (fast1 ? TJ_FAST1 : 0u) | (flat2 ? TJ_F2 : 0u) |
               (fast2 ? TJ_JFAST : 0u);
    if (emit) {
        const PathOut po = path_out<true, false>(A, path);
        uint32_t nlast = 2;
        if (!fast2) nlast = slow_join_summary(j.c3, j.c2, flat2, j.c1, P).vcount;
        j.base1 = po.id_base + S.vpre[b] - S.path_v[path];
        j.jbase = po.id_base + j.vcur - nlast;
    } else {
        // Ids of different joins differ, as they will; a sub-path of three points has one join.
        j.base1 = 0;
        j.jbase = j.n == 3 ? 0u : 1u << 28;
        j.vcur = 1u << 30;
    }
    return j;
}

// Threads take the sub-path ends of a tile of slots, packed so that the warps that run the caps are
// full: ends are a twentieth of the verbs of a drawing. Tiles are TAIL_TILE slots, and smaller ones
// in a batch too small for a tile per block, so that no thread runs two tails one after the other
// while other SMs are idle (1,000 paths of one line: 36 -> 21 us).
constexpr uint32_t TAIL_TILE = 1024, TAIL_THREADS = 128;
template <bool EMIT, bool REC>
__global__ void __launch_bounds__(TAIL_THREADS) tails_kernel(StrokeArgs A, StrokeVerbs S) {
    __shared__ uint32_t ends[TAIL_TILE];
    __shared__ uint32_t count;
    const uint32_t nv = batch_verbs(A);
    if (unfit(S, nv)) return;
    const uint32_t size = tile_size(nv, TAIL_THREADS, TAIL_TILE);
    for (uint32_t tile = blockIdx.x * size; tile < nv; tile += gridDim.x * size) {
        __syncthreads();
        if (threadIdx.x == 0) count = 0;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < size; i += blockDim.x) {
            const uint32_t v = tile + i;
            if (v < nv && is_end(S.kind[v] & KIND_MASK)) ends[atomicAdd(&count, 1u)] = v;
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) {
            const uint32_t v = ends[i], path = S.path[v];
            if (S.path_walk[path] || (EMIT && A.status[path] != LYON_OK)) continue;
            const StrokeParams P = make_params(A.options[A.num_options > 1 ? path : 0]);
            const TailJob j = tail_job<REC>(A, S, v, path, P, EMIT);
            uint32_t tv, ti;
            int st;
            const PathOut po = path_out<EMIT, REC>(A, path);
            tail_at<REC>(j, P, po, &tv, &ti, &st);
            if (EMIT) {
                if (st != LYON_OK || j.vcur + tv != S.vpre[v + 1] - S.path_v[path] ||
                    j.icur + ti != S.ipre[v + 1] - S.path_i[path])
                    A.status[path] = st != LYON_OK ? st : LYON_ERR_INTERNAL;
            } else {
                if (st != LYON_OK) leave_to_walk(S, path);
                S.vpre[v] = tv;
                S.ipre[v] = ti;
            }
        }
    }
}

// ---- 6. positions ------------------------------------------------------------------------------

// A verb's vertices and index words. The edge into a verb's first join is added here, from the join
// of the verb before it.
__device__ __forceinline__ void verb_counts(const StrokeArgs& A, const StrokeVerbs& S, uint32_t v,
                                            uint32_t nv, uint32_t& a, uint32_t& b) {
    a = b = 0;
    const int kind = v < nv ? (int)(S.kind[v] & KIND_MASK) : KIND_NONE;
    if ((is_segment(kind) || is_end(kind)) && !S.path_walk[S.path[v]]) {
        a = S.vpre[v];
        b = S.ipre[v];
        if (!A.widths && is_segment(kind) && (S.kind[v - 1] & KIND_MASK) != LYON_VERB_BEGIN) {
            const uint32_t f = S.flags[v];
            if (flags_nk(f) >= 2 || is_segment(S.kind[v + 1] & KIND_MASK))
                b += 3u * edge_count_flags(pj_from(S.join[v - 1]),
                                           f & VF_TOFIRST ? EF_SELF_EQ : 0u);
        }
    }
}

// Exclusive sums of the verbs' counts over the whole batch, in place (modulo 2^32: a position
// within a path is a difference of two): single-pass scan with decoupled look-back.
__global__ void __launch_bounds__(SCAN_THREADS) verb_scan_kernel(StrokeArgs A, StrokeVerbs S) {
    __shared__ uint32_t tile_s;
    __shared__ unsigned long long prefix_s[2];
    const uint32_t nv = batch_verbs(A);
    if (unfit(S, nv)) return;
    const uint32_t num_tiles = (nv + SCAN_TILE - 1) / SCAN_TILE;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) tile_s = atomicAdd(&S.words[5], 1u);
        __syncthreads();
        const uint32_t tile = tile_s;
        if (tile >= num_tiles) return;
        const uint32_t base = tile * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
        uint32_t va[SCAN_ITEMS], vb[SCAN_ITEMS];
        unsigned long long sa = 0, sb = 0;
#pragma unroll
        for (int i = 0; i < SCAN_ITEMS; ++i) {
            uint32_t a, b;
            verb_counts(A, S, base + i, nv, a, b);
            va[i] = a;
            vb[i] = b;
            sa += a;
            sb += b;
        }
        unsigned long long ta, tb;
        const unsigned long long ea = block_excl_scan(sa, &ta), eb = block_excl_scan(sb, &tb);
        if (threadIdx.x < 32)
            scan_publish(S.scan, num_tiles, tile, ta, tb, prefix_s,
                         reinterpret_cast<int*>(&S.words[1]));
        __syncthreads();
        uint32_t ra = (uint32_t)(prefix_s[0] + ea), rb = (uint32_t)(prefix_s[1] + eb);
#pragma unroll
        for (int i = 0; i < SCAN_ITEMS; ++i) {
            const uint32_t v = base + i;
            if (v < nv) {
                S.vpre[v] = ra;
                S.ipre[v] = rb;
            }
            ra += va[i];
            rb += vb[i];
            if (v + 1 == nv) {
                S.vpre[nv] = ra;
                S.ipre[nv] = rb;
            }
        }
    }
}

__global__ void __launch_bounds__(256) paths_kernel(StrokeArgs A, StrokeVerbs S) {
    const uint32_t v0 = A.verb_offsets[0], nv = batch_verbs(A);
    const bool none = unfit(S, nv);
    for (uint32_t path = blockIdx.x * blockDim.x + threadIdx.x; path < A.num_paths;
         path += gridDim.x * blockDim.x) {
        uint32_t vc = 0, ic = 0;
        if (!none) {
            const uint32_t s0 = A.verb_offsets[path] - v0, s1 = A.verb_offsets[path + 1] - v0;
            if (nv > 0) {
                const uint32_t pv = S.vpre[s0], pi = S.ipre[s0];
                vc = S.vpre[s1] - pv;
                ic = S.ipre[s1] - pi;
                S.path_v[path] = pv;
                S.path_i[path] = pi;
            }
            if (S.path_walk[path]) S.walk_list[atomicAdd(&S.words[2], 1u)] = path;
        }
        A.vtx_counts[path] = vc;
        A.idx_counts[path] = ic;
        A.status[path] = LYON_OK;
    }
}

// All that follows the verbs' counts, by one block: with VERBS their positions, then the paths'
// counts (paths_kernel), the index range per path, the paths' places and the totals (the kernels of
// scan.cu). For few paths these are short kernels one after another, of which the launches are most:
// five, with three fills of words before them, for which one path's call took 169 us and takes 157.
// (1,000 paths of 16 segments gain less than their spread from run to run.)
template <bool VERBS>
__global__ void __launch_bounds__(SCAN_THREADS) finish_kernel(StrokeArgs A, StrokeVerbs S,
                                                              StrokeFinish F) {
    __shared__ uint32_t failed_s;
    const uint32_t v0 = A.verb_offsets[0], nv = batch_verbs(A);
    const bool none = unfit(S, nv);
    if (threadIdx.x == 0) failed_s = 0;
    __syncthreads();
    if (VERBS && !none) {
        unsigned long long pa = 0, pb = 0;
        for (uint32_t at = 0; at < nv; at += SCAN_TILE) {
            const uint32_t base = at + threadIdx.x * SCAN_ITEMS;
            uint32_t va[SCAN_ITEMS], vb[SCAN_ITEMS];
            unsigned long long sa = 0, sb = 0;
#pragma unroll
            for (int i = 0; i < SCAN_ITEMS; ++i) {
                verb_counts(A, S, base + i, nv, va[i], vb[i]);
                sa += va[i];
                sb += vb[i];
            }
            unsigned long long ta, tb;
            const unsigned long long ea = block_excl_scan(sa, &ta), eb = block_excl_scan(sb, &tb);
            uint32_t ra = (uint32_t)(pa + ea), rb = (uint32_t)(pb + eb);
#pragma unroll
            for (int i = 0; i < SCAN_ITEMS; ++i) {
                if (base + i < nv) {
                    S.vpre[base + i] = ra;
                    S.ipre[base + i] = rb;
                }
                ra += va[i];
                rb += vb[i];
            }
            pa += ta;
            pb += tb;
        }
        if (threadIdx.x == 0 && nv > 0) {
            S.vpre[nv] = (uint32_t)pa;
            S.ipre[nv] = (uint32_t)pb;
        }
        __syncthreads();
    }
    unsigned long long pa = 0, pb = 0;
    for (uint32_t at = 0; at < A.num_paths; at += SCAN_THREADS) {
        const uint32_t path = at + threadIdx.x;
        uint32_t vc = 0, ic = 0;
        if (path < A.num_paths) {
            int32_t status = LYON_OK;
            if (!none) {
                const uint32_t s0 = A.verb_offsets[path] - v0, s1 = A.verb_offsets[path + 1] - v0;
                if (nv > 0) {
                    const uint32_t pv = S.vpre[s0], pi = S.ipre[s0];
                    vc = S.vpre[s1] - pv;
                    ic = S.ipre[s1] - pi;
                    S.path_v[path] = pv;
                    S.path_i[path] = pi;
                }
                if (S.path_walk[path]) S.walk_list[atomicAdd(&S.words[2], 1u)] = path;
            }
            if (vc > 0 && F.vertex_offset + vc - 1 > F.max_index) {
                status = LYON_ERR_TOO_MANY_VERTICES;
                vc = ic = 0;
                atomicAdd(&failed_s, 1u);
            }
            A.vtx_counts[path] = vc;
            A.idx_counts[path] = ic;
            A.status[path] = status;
        }
        unsigned long long ta, tb;
        const unsigned long long ea = block_excl_scan((unsigned long long)vc, &ta);
        const unsigned long long eb = block_excl_scan((unsigned long long)ic, &tb);
        if (path < A.num_paths) {
            F.vtx_offsets[path] = pa + ea;
            F.idx_offsets[path] = pb + eb;
        }
        pa += ta;
        pb += tb;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        F.vtx_offsets[A.num_paths] = pa;
        F.idx_offsets[A.num_paths] = pb;
        F.words[0] = 0;
        F.words[1] = failed_s;
        F.host[0] = pa;
        F.host[1] = pb;
        F.host[2] = (uint64_t)failed_s << 32;
        const volatile uint32_t* w = S.words;
        F.host[3] = (uint64_t)w[0] | ((uint64_t)w[1] << 32);
        F.host[4] = (uint64_t)w[2] | ((uint64_t)w[3] << 32);
    }
}

// ---- runs of flattening-step joins ---------------------------------------------------------------
struct RunSlot {
    UnitSmem u;
    float2* vout;        // where the run's vertices go
    void* iout;          // where the run's indices go (the edge into its first join first)
    float hw;
    uint32_t id;         // id of its first vertex
    uint32_t pfn, pfp, edge_words;  // the edge into its first join: ids, index words
    float adv;           // the advancement before it (records)
};
struct RunSmem {
    RunSlot unit[WIN_UNITS];
    PointSmem pt;
};

// Word w of the indices of a run of edges between flattening-step joins, six per edge:
// (neg', pos', pos), (neg', pos, neg) with pos = first + 2 * edge, neg = pos + 1 and the previous
// join's pos' = pos - 2, neg' = pos - 1 (add_edge_triangles, stroke.rs:1869-1904).
__device__ __forceinline__ uint32_t run_index(uint32_t first, uint32_t e, uint32_t c) {
    // c:  0   1   2   3   4   5
    //    -1  -2   0  -1   0  +1   (stored + 2)
    return first + 2u * e + ((0x321201u >> (4u * c)) & 0xFu) - 2u;
}

// The pattern of run_index over 64 edges (384 words: whole numbers of edges and of 16-byte quads),
// once for every place a 16-byte boundary can have in it, so that a quad of indices is one load
// from shared memory and four additions. (Worked out per word it took as many instructions as the
// vertices' samples.)
constexpr uint32_t PATTERN = 384;
struct IndexPattern {
    int4 quad[4][PATTERN / 4];  // quad q of pattern h: words h + 4 q .. h + 4 q + 3, less the first id
};
__device__ __forceinline__ void make_pattern(IndexPattern& p) {
    for (uint32_t i = threadIdx.x; i < 4 * PATTERN; i += blockDim.x) {
        const uint32_t h = i / PATTERN, w = h + i % PATTERN;
        reinterpret_cast<int*>(p.quad[h])[i % PATTERN] = (int)run_index(0u, w / 6u, w % 6u);
    }
    __syncthreads();
}

__device__ __forceinline__ void write_run_indices(uint32_t* dst, uint32_t words, uint32_t first,
                                                  const IndexPattern& p, int lane) {
    const uint32_t mis = (uint32_t)((reinterpret_cast<uintptr_t>(dst) & 15u) / 4u);
    const uint32_t head = min(words, (4u - mis) & 3u);
    const uint32_t quads = (words - head) / 4u, tail = head + quads * 4u;
    if ((uint32_t)lane < head) dst[lane] = run_index(first, 0u, (uint32_t)lane);
    int4* out = reinterpret_cast<int4*>(dst + head);
    const int4* pat = p.quad[head];
    uint32_t base = first;  // 64 edges: 96 quads, 128 ids
    for (uint32_t q0 = 0; q0 < quads; q0 += PATTERN / 4, base += 128u) {
#pragma unroll
        for (uint32_t j = 0; j < 3; ++j) {
            const uint32_t q = j * 32u + (uint32_t)lane;
            if (q0 + q < quads) {
                int4 x = pat[q];
                x.x += (int)base;
                x.y += (int)base;
                x.z += (int)base;
                x.w += (int)base;
                out[q0 + q] = x;
            }
        }
    }
    if (tail + (uint32_t)lane < words) {
        const uint32_t w = tail + (uint32_t)lane;
        dst[w] = run_index(first, w / 6u, w % 6u);
    }
}
__device__ __forceinline__ void write_run_indices(uint16_t* dst, uint32_t words, uint32_t first,
                                                  const IndexPattern&, int lane) {
    const uint32_t mis = (uint32_t)((reinterpret_cast<uintptr_t>(dst) & 15u) / 2u);
    const uint32_t head = min(words, (8u - mis) & 7u);
    const uint32_t quads = (words - head) / 8u, tail = head + quads * 8u;
    if ((uint32_t)lane < head) dst[lane] = (uint16_t)run_index(first, lane / 6u, lane % 6u);
    for (uint32_t q = (uint32_t)lane; q < quads; q += 32) {
        const uint32_t w = head + q * 8u;
        uint32_t e = w / 6u, c = w - 6u * e;
        uint32_t x[8];
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) {
            x[i] = run_index(first, e, c);
            if (++c == 6u) {
                c = 0;
                ++e;
            }
        }
        *reinterpret_cast<uint4*>(dst + w) =
            make_uint4((x[0] & 0xFFFFu) | (x[1] << 16), (x[2] & 0xFFFFu) | (x[3] << 16),
                       (x[4] & 0xFFFFu) | (x[5] << 16), (x[6] & 0xFFFFu) | (x[7] << 16));
    }
    if (tail + (uint32_t)lane < words) {
        const uint32_t w = tail + (uint32_t)lane;
        dst[w] = (uint16_t)run_index(first, w / 6u, w % 6u);
    }
}

// Lane = point: tangent of the edge into the point, normal and two vertices of the join at the point
// before, 16 bytes a lane; the indices of a run are a formula of their position and leave as
// 16-byte stores too. Bound by instruction issue (the divisions and square roots of the normals:
// IEEE, as lyon's) and the stores. Records take a sum over the points besides, one addition after
// another as lyon's advancement does: 32 for 32 points.
template <bool REC>
__global__ void __launch_bounds__(WIN_WARPS * 32) runs_kernel(StrokeArgs A, StrokeVerbs S) {
    extern __shared__ __align__(16) unsigned char run_smem[];
    const int lane = threadIdx.x & 31;
    IndexPattern& pattern = *reinterpret_cast<IndexPattern*>(run_smem);
    RunSmem& sm = reinterpret_cast<RunSmem*>(run_smem + sizeof(IndexPattern))[threadIdx.x >> 5];
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t nv = batch_verbs(A);
    if (nv > S.cap) return;
    const uint32_t W = window_verbs(nv, nwarps);
    make_pattern(pattern);
    for (uint32_t w0 = warp * W; w0 < nv; w0 += nwarps * W) {
        // ---- the window's units ----
        const uint32_t v = w0 + (uint32_t)lane;
        Unit a, b;
        a.m = b.m = 0;
        VerbOut oa, ob;  // where each unit's run goes
        float hw = 0.0f;
        V2 c1 = V2{0.0f, 0.0f};
        if ((uint32_t)lane < W && v < nv) {
            const int kind = S.kind[v] & KIND_MASK;
            const uint32_t path = S.path[v];
            if ((kind == LYON_VERB_QUADRATIC_TO || kind == LYON_VERB_CUBIC_TO) &&
                !(S.flags[v] & VF_IRR) && !S.path_walk[path] && A.status[path] == LYON_OK) {
                const StrokeParams P = make_params(A.options[A.num_options > 1 ? path : 0]);
                const uint32_t flags = S.flags[v];
                verb_units(kind, S.rec[v], A.points, P.tolerance, flags,
                           flags & VF_TWO ? S.cut[v] : 0u, a, b);
                hw = P.hw;
                c1 = last_kept(S, A.points, v - 1);
                verb_out<REC>(A, S, v, path, oa);
                ob = oa;
                if (REC && b.m > 0) ob.adv = S.adv[v].x;
                pass_run(ob, a.m - 1u);
                const uint32_t va = ob.vo, ia = ob.io;
                uint32_t vb = 0, ib = 0;
                if (b.m > 0) {
                    // Past the join between the two.
                    const uint32_t j = S.split[v];
                    const uint32_t e = ob.edge ? edge_count_flags(
                                                     ob.pfn == ob.pfp ? EF_SELF_EQ : 0u, pj_to(j))
                                               : 0u;
                    ob.pfn = ob.po.id_base + ob.vo + pj_neg(j);
                    ob.pfp = ob.po.id_base + ob.vo + pj_pos(j);
                    ob.vo += pj_vertices(j);
                    ob.io += 3u * (e + pj_tris(j));
                    ob.edge = true;
                    VerbOut past = ob;
                    pass_run(past, b.m - 1u);
                    vb = past.vo;
                    ib = past.io;
                }
                // What the count phase reserved bounds every write.
                if (max(va, vb) > oa.po.vmax || max(ia, ib) > oa.po.imax) {
                    A.status[path] = LYON_ERR_INTERNAL;
                    a.m = b.m = 0;
                }
            }
        }
        const bool ra = a.m >= 2, rb = b.m >= 2;  // runs of this lane
        const uint32_t mask_a = __ballot_sync(FULL, ra), mask_b = __ballot_sync(FULL, rb);
        if ((mask_a | mask_b) == 0) continue;
        const uint32_t below = (1u << lane) - 1u;
        const uint32_t slot = __popc(mask_a & below) + __popc(mask_b & below);
        const uint32_t nunits = __popc(mask_a) + __popc(mask_b);
        const uint32_t steps = (ra ? a.m : 0u) + (rb ? b.m : 0u);
        uint32_t incl = steps;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t up = __shfl_up_sync(FULL, incl, d);
            if (lane >= d) incl += up;
        }
        const uint32_t total = __shfl_sync(FULL, incl, 31);
        const uint32_t excl = incl - steps;
        auto lay_out = [&](RunSlot& r, const Unit& x, V2 from, const VerbOut& o, uint32_t first) {
            lay_out_unit(r.u, x, from, first);
            r.hw = hw;
            r.vout = REC ? reinterpret_cast<float2*>(o.po.rout + o.vo) : o.po.vout + o.vo;
            r.adv = o.adv;
            r.iout = o.po.bits == 16 ? (void*)((uint16_t*)o.po.iout + o.io)
                                     : (void*)((uint32_t*)o.po.iout + o.io);
            r.id = o.po.id_base + o.vo;
            r.pfn = o.pfn;
            r.pfp = o.pfp;
            r.edge_words = 3u * edge_into_step(o);
        };
        if (ra) lay_out(sm.unit[slot], a, c1, oa, excl);
        if (rb) lay_out(sm.unit[slot + (ra ? 1u : 0u)], b, a.to, ob, excl + (ra ? a.m : 0u));
        __syncwarp();
        // ---- vertices ----
        V2 q = V2{0.0f, 0.0f}, nt = V2{0.0f, 0.0f};
        float sum = 0.0f;  // the advancement at the last point (records)
        for (uint32_t r0 = 0; r0 < total; r0 += WIN_ROUND) {
            const uint32_t rn = min(WIN_ROUND, total - r0);
            fill_points(sm.pt, &sm.unit[0].u, sizeof(RunSlot), nunits, r0, rn, lane);
            for (uint32_t cb = 0; cb < rn; cb += 32) {
                const uint32_t at = cb + (uint32_t)lane;
                const uint32_t i = min(at, rn - 1u);
                const RunSlot& r = sm.unit[sm.pt.owner[i]];
                const uint32_t k = r0 + i - r.u.excl + 1u, m = r.u.m_cubic >> 1;
                const V2 old_q = q, old_t = nt;
                q = unit_point(r.u, k, sm.pt.t[i]);
                V2 qp = V2{from_left(q.x, old_q.x, lane), from_left(q.y, old_q.y, lane)};
                if (k == 1u) {
                    const float4 e = r.u.c1_to;
                    qp = V2{e.x, e.y};
                }
                const V2 ne = q - qp;
                const float len = vlength(ne);
                nt = ne / len;
                float adv = 0.0f;  // at the point before, where the join is
                if constexpr (REC) {
                    const uint32_t starts = __ballot_sync(FULL, k == 1u);
#pragma unroll
                    for (uint32_t j = 0; j < 32; ++j) {
                        if ((starts >> j) & 1u) sum = __shfl_sync(FULL, r.adv, (int)j);
                        if ((uint32_t)lane == j) adv = sum;
                        sum = sum + __shfl_sync(FULL, len, (int)j);
                    }
                }
                const V2 pt = V2{from_left(nt.x, old_t.x, lane), from_left(nt.y, old_t.y, lane)};
                const float rhw = r.hw;
                const V2 nrm = compute_normal(pt, nt);
                const V2 pn = qp + nrm * rhw, nn = qp - nrm * rhw;
                // The vertices (pn, nn) of the join at point k - 1 start at 2 (k - 2). When that is
                // no 16-byte boundary, a lane writes its left neighbour's nn with its own pn.
                const V2 ln = V2{__shfl_up_sync(FULL, nn.x, 1), __shfl_up_sync(FULL, nn.y, 1)};
                if (REC) {
                    if (at < rn && k > 1u) {
                        float2* dst = r.vout + 6u * (k - 2u);
                        if ((reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
                            float4* d = reinterpret_cast<float4*>(dst);
                            d[0] = make_float4(pn.x, pn.y, nrm.x, nrm.y);
                            d[1] = make_float4(adv, __uint_as_float((uint32_t)SP), nn.x, nn.y);
                            d[2] = make_float4(-nrm.x, -nrm.y, adv, __uint_as_float((uint32_t)SN));
                        } else {
                            dst[0] = make_float2(pn.x, pn.y);
                            dst[1] = make_float2(nrm.x, nrm.y);
                            dst[2] = make_float2(adv, __uint_as_float((uint32_t)SP));
                            dst[3] = make_float2(nn.x, nn.y);
                            dst[4] = make_float2(-nrm.x, -nrm.y);
                            dst[5] = make_float2(adv, __uint_as_float((uint32_t)SN));
                        }
                    }
                } else if (at < rn && k > 1u) {
                    float2* dst = r.vout + 2u * (k - 2u);
                    if ((reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
                        *reinterpret_cast<float4*>(dst) = make_float4(pn.x, pn.y, nn.x, nn.y);
                    } else {
                        if (lane > 0 && k > 2u) {
                            *reinterpret_cast<float4*>(dst - 1) = make_float4(ln.x, ln.y, pn.x, pn.y);
                        } else {
                            dst[0] = make_float2(pn.x, pn.y);
                        }
                        if (lane == 31 || at + 1u == rn || k == m)
                            dst[1] = make_float2(nn.x, nn.y);
                    }
                }
            }
            __syncwarp();
        }
        // ---- indices ----
        for (uint32_t u = 0; u < nunits; ++u) {
            const RunSlot& r = sm.unit[u];
            const uint32_t ew = r.edge_words, words = 6u * ((r.u.m_cubic >> 1) - 2u), id = r.id;
            // The edge into the first join: (pfn, pfp, pos), (pfn, pos, neg); without the first
            // when pfn == pfp.
            uint32_t x = 0;
            if ((uint32_t)lane < ew) {
                const uint32_t c = (uint32_t)lane + (6u - ew);
                x = c == 0 || c == 3 ? r.pfn : c == 1 ? r.pfp : c == 5 ? id + 1u : id;
            }
            if (A.index_bits == 16) {
                uint16_t* d = (uint16_t*)r.iout;
                if ((uint32_t)lane < ew) d[lane] = (uint16_t)x;
                write_run_indices(d + ew, words, id + 2u, pattern, lane);
            } else {
                uint32_t* d = (uint32_t*)r.iout;
                if ((uint32_t)lane < ew) d[lane] = x;
                write_run_indices(d + ew, words, id + 2u, pattern, lane);
            }
        }
        __syncwarp();
    }
}

constexpr size_t RUN_SMEM = sizeof(IndexPattern) + WIN_WARPS * sizeof(RunSmem);
static_assert(WIN_WARPS * sizeof(WalkSmem) <= 48 * 1024 && RUN_SMEM <= 48 * 1024,
              "shared memory of the window kernels");

uint32_t grid_for(uint32_t items, uint32_t per_block, int num_sms, uint32_t waves) {
    const uint32_t sms = (uint32_t)(num_sms > 0 ? num_sms : 1);
    const uint32_t need = (items + per_block - 1) / per_block;
    // At least a block per SM: the hint may be short of what the batch holds.
    return need < sms ? sms : need > sms * waves ? sms * waves : need;
}

}  // namespace

cudaError_t launch_stroke_verbs_count(const StrokeArgs& a, const StrokeVerbs& v,
                                      uint32_t verbs_hint, int num_sms, const SideStreams& side,
                                      const StrokeFinish* finish, cudaStream_t s) {
    const uint32_t n = a.num_paths;
    cudaMemsetAsync(v.words, 0, v.clear_bytes, s);
    const uint32_t by_path = grid_for(n, 8, num_sms, 8);
    const uint32_t by_verb = grid_for(verbs_hint, 256, num_sms, 8);
    prepare_kernel<<<by_path, 256, 0, s>>>(a, v);
    turns_kernel<<<grid_for(verbs_hint, TURN_TILE, num_sms, 4), 256, 0, s>>>(a, v);
    walk_kernel<<<grid_for(verbs_hint, WIN_WARPS, num_sms, 8), WIN_WARPS * 32,
                  WIN_WARPS * sizeof(WalkSmem), s>>>(a, v);
    drops_kernel<<<grid_for(0, 128, num_sms, 1), 128, 0, s>>>(a, v);
    const bool advance = a.vertex_attrs && !a.widths && n <= STROKE_ADVANCE_EARLY;
    if (advance) launch_stroke_advance(a, v, num_sms, side, s);
    if (a.widths) {
        launch_stroke_steps_count(a, v, verbs_hint, num_sms, side, s);
    } else {
        // Tails read the points beside the sub-paths' ends and nothing of the joins.
        const cudaStream_t t = side.fork(0, s);
        tails_kernel<false, false><<<grid_for(verbs_hint, TAIL_TILE, num_sms, 16), 128, 0, t>>>(a, v);
        extra_count_kernel<<<grid_for(verbs_hint / 8, 128, num_sms, 8), 128, 0, s>>>(a, v);
        joins_count_kernel<<<by_verb, 256, 0, s>>>(a, v);
        side.join(0, s);
        note_launches(3);
    }
    note_launches(5);
    // One tile of verbs is summed by the block that finishes; more by as many blocks.
    const bool one_tile = finish && verbs_hint <= SCAN_TILE;
    if (one_tile) {
        finish_kernel<true><<<1, SCAN_THREADS, 0, s>>>(a, v, *finish);
    } else {
        verb_scan_kernel<<<grid_for(verbs_hint, SCAN_TILE, num_sms, 4), SCAN_THREADS, 0, s>>>(a, v);
        if (finish) {
            finish_kernel<false><<<1, SCAN_THREADS, 0, s>>>(a, v, *finish);
        } else {
            paths_kernel<<<grid_for(n, 256, num_sms, 8), 256, 0, s>>>(a, v);
        }
        note_launches(1);
    }
    if (advance) join_stroke_advance(side, s);
    return cudaGetLastError();
}

template <bool REC>
static void launch_verbs_emit(const StrokeArgs& a, const StrokeVerbs& v, uint32_t verbs_hint, bool runs,
                              int num_sms, const SideStreams& side, cudaStream_t s) {
    // The three write different parts of the output; joins and tails are short of warps and of
    // threads that agree, and fill the gaps of the runs.
    const cudaStream_t j = side.fork(0, s), t = side.fork(1, s);
    if (runs) {
        runs_kernel<REC><<<grid_for(verbs_hint, WIN_WARPS, num_sms, 8), WIN_WARPS * 32, RUN_SMEM,
                           s>>>(a, v);
        note_launches(1);
    }
    // (joins and tails are the shorter ones of a small batch, and share a stream: 1,000 paths of 16
    // segments take 12 and 42 us there, the runs 58, the verbs apart 79)
    extra_emit_kernel<REC><<<grid_for(verbs_hint / 8, 128, num_sms, 8), 128, 0, j>>>(a, v);
    joins_emit_kernel<REC><<<grid_for(verbs_hint, 256, num_sms, 8), 256, 0, t>>>(a, v);
    tails_kernel<true, REC><<<grid_for(verbs_hint, TAIL_TILE, num_sms, 16), 128, 0, t>>>(a, v);
    note_launches(3);
    side.join(0, s);
    side.join(1, s);
}

cudaError_t launch_stroke_verbs_emit(const StrokeArgs& a, const StrokeVerbs& v,
                                     uint32_t verbs_hint, bool runs, int num_sms,
                                     const SideStreams& side, cudaStream_t s) {
    if (a.widths || a.sources) return launch_stroke_steps_emit(a, v, verbs_hint, num_sms, side, s);
    if (a.vertex_attrs) {
        if (a.num_paths > STROKE_ADVANCE_EARLY) {
            launch_stroke_advance(a, v, num_sms, side, s);
            join_stroke_advance(side, s);
        }
        launch_verbs_emit<true>(a, v, verbs_hint, runs, num_sms, side, s);
    } else {
        launch_verbs_emit<false>(a, v, verbs_hint, runs, num_sms, side, s);
    }
    return cudaGetLastError();
}

}  // namespace lg
