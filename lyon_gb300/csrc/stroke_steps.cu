// stroke_steps.cu — lyon's sequential stroke stepper, one verb per thread.
//
// Variable line width and vertex sources want the stepper itself
// (stroke_seq.cuh, stroke_core.cuh). Its state is short: the last two points with their sides,
// ids and advancement. So a thread can step one verb by itself once it has that state, which it
// gets by stepping the last four kept points before the verb first, without output (a point's
// sides come from its neighbours, and theirs, which matter to a skip test only, from the next).
// stroke_verbs.cu has said which points are kept; the advancement, a running f32 sum over the whole
// path, is worked out beforehand (advance_kernel) at the points a thread may start from.
//
// With a fixed width the count phase of stroke_verbs.cu has the counts, and has ruled out all that
// would make the state depend on more. With a variable width the stepper counts as well, and the
// claim is checked: a hash of the state a thread started its verb with has to equal the one the
// thread of the verb before ended with, over all verbs of the path, and each sub-path's end has to
// leave the advancement that the next one started with, or the path is stroked by one thread as a
// whole (stroke_seq.cu), as are the paths that stroke_verbs.cu leaves out. (A clipped miter moves
// side points of the joins after it, so those paths usually go that way.)
//
// The advancement kernels also serve attribute records, which stroke_verbs.cu writes run by run.
//
// Bound by instruction issue with 9 to 12 of a warp's 32 lanes at work (curves of different lengths,
// general joins among flattening steps). Measured, whole calls on one GB300, against one thread
// per path: variable width on 10,001 curve paths 159 -> 6.9 ms, vertex sources and two custom values
// on 9,999 paths 82 -> 2.3 ms.
#include "stroke_seq.cuh"
#include "stroke_verbs.cuh"

namespace lg {
namespace {

// The four advancements kept per verb: those of its last four kept points (.w: the last one).
__device__ __forceinline__ float4* advancements(const StrokeVerbs& S) { return S.adv; }
__device__ __forceinline__ float advancement_back(const StrokeVerbs& S, uint32_t v, uint32_t back) {
    return reinterpret_cast<const float*>(advancements(S) + v)[3u - back];
}
// The state hashes (variable width): the one a verb started with and the one it ended with.
__device__ __forceinline__ ulonglong2* state_hashes(const StrokeVerbs& S) {
    return reinterpret_cast<ulonglong2*>(S.lasts);
}

// ---- advancement -------------------------------------------------------------------------------
// lyon's advancement is a running f32 sum of edge lengths (stroke.rs:1546-1550, 1657-1662,
// 1759-1771), so the lengths are worked out at once, lane = point, and added one after the other.
struct AdvanceState {
    float adv, start;  // at the last kept point; where the next sub-path starts
    uint32_t kept;
};

// Verbs that are no run of points (every lane of a warp alike): a sub-path's begin and end, and an
// irregular verb's merge chain.
__device__ __forceinline__ void advance_special(const StrokeArgs& A, const StrokeVerbs& S,
                                                uint32_t v, int kind, const StrokeParams& P,
                                                AdvanceState& st, int lane) {
    float* out = reinterpret_cast<float*>(advancements(S) + v);
    if (kind == LYON_VERB_BEGIN) {
        st.adv = st.start;
        st.kept = 1;
        if (lane == 0) out[3] = st.adv;
    } else if (is_end(kind)) {
        // end_with_caps carries the last advancement on (stroke.rs:1359). (With a variable width
        // step_verb checks it.)
        if (st.kept >= 2 && !(kind == LYON_VERB_CLOSE && st.kept > 2)) st.start = st.adv;
    } else if (is_segment(kind)) {
        const uint32_t flags = S.flags[v];
        Unit a, b;
        verb_units(kind, S.rec[v], A.points, P.tolerance, flags & VF_TURN,
                   flags & VF_TURN ? S.cut[v] : 0u, a, b);
        V2 last = last_kept(S, A.points, v - 1);
        float before = st.adv;  // at the last kept point but one
        for (uint32_t u = 0; u < (b.m ? 2u : 1u); ++u) {
            float t = a.t0;
            for (uint32_t k = 1; k <= a.m; ++k) {
                V2 q = a.to;
                if (k < a.m) {
                    t = t + a.s;
                    q = poly_sample(a.p, t);
                }
                if (too_close(last, q, P.merge_threshold)) continue;
                before = st.adv;
                st.adv = st.adv + vlength(q - last);
                last = q;
                ++st.kept;
            }
            a = b;
        }
        if (lane == 0) {
            out[2] = before;
            out[3] = st.adv;
        }
    }
}

// Calls use(i, count, len, edges, first) for the verb's edges 32 at a time: lane's edge i (0-based;
// >= the verb's edges: none) and its length, how many edges the verb has and how many of them are
// its first run's (0: there is one run only). Returns the number of edges.
template <class F>
__device__ __forceinline__ uint32_t verb_edges(const StrokeArgs& A, const StrokeVerbs& S,
                                               uint32_t v, int kind, const StrokeParams& P,
                                               int lane, F use) {
    const uint32_t flags = S.flags[v];
    Unit a, b;
    verb_units(kind, S.rec[v], A.points, P.tolerance, flags, flags & VF_TWO ? S.cut[v] : 0u, a, b);
    V2 last = last_kept(S, A.points, v - 1);
    const uint32_t M = a.m + b.m, first = b.m ? a.m : 0u;
    uint32_t before = 0;
    for (uint32_t u = 0; u < (b.m ? 2u : 1u); ++u) {
        uint32_t tk = 0;
        float t0 = a.t0;
        for (uint32_t k0 = 1; k0 <= a.m; k0 += 32) {
            const uint32_t cnt = min(32u, a.m - k0 + 1u), kk = min(k0 + (uint32_t)lane, a.m);
            const float t = accumulate_t_from(a.s, tk, t0, kk);
            const V2 q = kk == a.m ? a.to : poly_sample(a.p, t);
            V2 p = V2{__shfl_up_sync(FULL, q.x, 1), __shfl_up_sync(FULL, q.y, 1)};
            if (lane == 0) p = last;
            use((uint32_t)lane < cnt ? before + kk - 1u : M, cnt, vlength(q - p), M, first);
            last = V2{__shfl_sync(FULL, q.x, (int)cnt - 1), __shfl_sync(FULL, q.y, (int)cnt - 1)};
            tk = k0 + cnt - 1u;
            t0 = __shfl_sync(FULL, t, (int)cnt - 1);
        }
        before = a.m;
        a = b;
    }
    return M;
}

// Running f32 sums over four-point words of shared memory, one addition after another: sums[i] =
// sums[i - 1] + lengths[i], from `adv`. Every lane runs it, lane 0 writes. A word is loaded while the
// one before it is added.
__device__ __forceinline__ float running_sums(const float4* lengths, float4* sums, uint32_t words,
                                              float adv, int lane) {
    float4 next = words > 0 ? lengths[0] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
    for (uint32_t w = 0; w < words; ++w) {
        float4 x = next;
        if (w + 1u < words) next = lengths[w + 1u];
        x.x = adv + x.x;
        x.y = x.x + x.y;
        x.z = x.y + x.z;
        x.w = x.z + x.w;
        adv = x.w;
        if (lane == 0) sums[w] = x;
    }
    return adv;
}

// Paths of more verbs than this are taken by blocks (below), the others by warps; so are long ones
// that are nearly all lines (a point a verb, or fewer): a warp takes 32 lines at once.
constexpr uint32_t ADVANCE_LONG = 64;
__device__ __forceinline__ bool advance_by_block(const StrokeArgs& A, uint32_t path,
                                                 uint32_t verbs) {
    const uint32_t points = A.point_offsets[path + 1] - A.point_offsets[path];
    return verbs > ADVANCE_LONG && points > verbs + verbs / 16u;
}

// The advancement at edge e's end, of M, where it is one of the last four; with `first` (the edges of
// the first of two runs) the one between the runs takes the first place.
__device__ __forceinline__ void keep_advancement(float* out, uint32_t e, uint32_t M, uint32_t first,
                                                 float adv) {
    if (e < M && e + (first ? 3u : 4u) >= M) out[4u - (M - e)] = adv;
    if (first && e + 1u == first) out[0] = adv;
}

// Warp per path. Bound by the sum's chain, 32 additions for 32 points, which run on words of shared
// memory (a shuffle per addition took 0.76 ms for 20,000 paths, this 0.62).
__global__ void __launch_bounds__(128) advance_kernel(StrokeArgs A, StrokeVerbs S) {
    __shared__ float4 lengths[4][8], sums[4][8];
    const int lane = threadIdx.x & 31;
    float4* const len4 = lengths[threadIdx.x >> 5];
    float4* const sum4 = sums[threadIdx.x >> 5];
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    if (unfit(S, batch_verbs(A))) return;
    const uint32_t v0 = A.verb_offsets[0];
    float* out = reinterpret_cast<float*>(advancements(S));
    const bool runs = !A.widths && !A.sequential;  // records: written run by run (stroke_verbs.cu)
    for (uint32_t path = warp; path < A.num_paths; path += nwarps) {
        const uint32_t s0 = A.verb_offsets[path] - v0, s1 = A.verb_offsets[path + 1] - v0;
        if (advance_by_block(A, path, s1 - s0) || S.path_walk[path]) continue;
        const StrokeParams P = make_params(A.options[A.num_options > 1 ? path : 0]);
        AdvanceState st{0.0f, 0.0f, 0};
        for (uint32_t base = s0; base < s1; base += 32) {
            const uint32_t n = min(32u, s1 - base);
            const int kind = (uint32_t)lane < n ? S.kind[base + lane] & KIND_MASK : KIND_NONE;
            const uint32_t lines = __ballot_sync(FULL, kind == LYON_VERB_LINE_TO);
            for (uint32_t i = 0; i < n; ++i) {
                const uint32_t v = base + i;
                const int k = __shfl_sync(FULL, kind, (int)i);
                // Lines in a row: lane = verb.
                const uint32_t others = ~lines >> i;
                const uint32_t row = others ? (uint32_t)__ffs((int)others) - 1u : 32u - i;
                if (row > 1u) {
                    const uint32_t u = v + (uint32_t)lane;
                    float len = 0.0f;
                    if ((uint32_t)lane < row)
                        len = vlength(end_point(S, A.points, u) - last_kept(S, A.points, u - 1));
                    reinterpret_cast<float*>(len4)[lane] = len;
                    __syncwarp();
                    st.adv = running_sums(len4, sum4, (row + 3u) / 4u, st.adv, lane);
                    __syncwarp();
                    if ((uint32_t)lane < row)
                        out[4 * (size_t)u + 3] = reinterpret_cast<const float*>(sum4)[lane];
                    __syncwarp();
                    st.kept += row;
                    i += row - 1u;
                    continue;
                }
                if (!is_segment(k) || (S.flags[v] & VF_IRR)) {
                    advance_special(A, S, v, k, P, st, lane);
                    continue;
                }
                st.kept += verb_edges(A, S, v, k, P, lane, [&](uint32_t e, uint32_t cnt, float len,
                                                               uint32_t M, uint32_t m1) {
                    reinterpret_cast<float*>(len4)[lane] = (uint32_t)lane < cnt ? len : 0.0f;
                    __syncwarp();
                    st.adv = running_sums(len4, sum4, (cnt + 3u) / 4u, st.adv, lane);
                    __syncwarp();
                    keep_advancement(out + 4 * (size_t)v, e, M, runs ? m1 : 0u,
                                     reinterpret_cast<const float*>(sum4)[lane]);
                    __syncwarp();
                });
            }
        }
    }
}

// Block per long path: the lengths of a window of verbs by all its warps, then the sums over them by
// one (one warp for both took 1.9 ms for a path of 35,000 points; with the four places of each verb
// kept during the sum 0.93 ms, taken from the stored sums afterwards, lane = verb, 0.74).
constexpr uint32_t ADVANCE_ROOM = 4096;
__global__ void __launch_bounds__(256) advance_long_kernel(StrokeArgs A, StrokeVerbs S) {
    __shared__ float4 room[ADVANCE_ROOM / 4], sums[ADVANCE_ROOM / 4];
    __shared__ uint32_t first[33];
    __shared__ int kinds[32];
    __shared__ uint32_t split[32];  // edges of the first of two runs, else 0
    __shared__ uint32_t window, num_long;
    __shared__ uint16_t longs[256];
    float* len = reinterpret_cast<float*>(room);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (unfit(S, batch_verbs(A))) return;
    const uint32_t v0 = A.verb_offsets[0];
    float* out = reinterpret_cast<float*>(advancements(S));
    const bool runs = !A.widths && !A.sequential;
    // A block looks through a tile of paths at once, and takes the long ones.
    const uint32_t size = tile_size(A.num_paths, 1u, 256u);
    for (uint32_t tile = blockIdx.x * size; tile < A.num_paths; tile += gridDim.x * size) {
        __syncthreads();
        if (threadIdx.x == 0) num_long = 0;
        __syncthreads();
        if (threadIdx.x < size && tile + threadIdx.x < A.num_paths) {
            const uint32_t p = tile + threadIdx.x;
            if (advance_by_block(A, p, A.verb_offsets[p + 1] - A.verb_offsets[p]) && !S.path_walk[p])
                longs[atomicAdd(&num_long, 1u)] = (uint16_t)threadIdx.x;
        }
        __syncthreads();
        for (uint32_t at = 0; at < num_long; ++at) {
            const uint32_t path = tile + longs[at];
            const uint32_t s0 = A.verb_offsets[path] - v0, s1 = A.verb_offsets[path + 1] - v0;
            const StrokeParams P = make_params(A.options[A.num_options > 1 ? path : 0]);
            AdvanceState st{0.0f, 0.0f, 0};
            for (uint32_t base = s0; base < s1;) {
                __syncthreads();
                if (warp == 0) {
                    // The window's verbs, their points rounded up to 16-byte words.
                    const uint32_t v = base + (uint32_t)lane;
                    int k = v < s1 ? S.kind[v] & KIND_MASK : KIND_NONE;
                    uint32_t m = 0, m1 = 0;
                    if (is_segment(k)) {
                        const uint32_t flags = S.flags[v];
                        if (flags & VF_IRR) {
                            k |= 8;
                        } else {
                            Unit a, b;
                            verb_units(k, S.rec[v], A.points, P.tolerance, flags,
                                       flags & VF_TWO ? S.cut[v] : 0u, a, b);
                            m = a.m + b.m;
                            if (runs && b.m) m1 = a.m;
                        }
                    }
                    split[lane] = m1;
                    uint32_t incl = (m + 3u) & ~3u;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t up = __shfl_up_sync(FULL, incl, o);
                        if (lane >= o) incl += up;
                    }
                    first[lane] = incl - ((m + 3u) & ~3u);
                    kinds[lane] = k | (int)(m << 4);
                    const uint32_t fit = __ballot_sync(FULL, incl <= ADVANCE_ROOM && v < s1);
                    if (lane == 0) window = (uint32_t)__popc(fit);
                }
                __syncthreads();
                const uint32_t n = window;
                for (uint32_t i = (uint32_t)warp; i < n; i += blockDim.x / 32) {
                    const int k = kinds[i] & 15;
                    if (!is_segment(k)) continue;
                    verb_edges(A, S, base + i, k, P, lane,
                               [&](uint32_t e, uint32_t, float x, uint32_t M, uint32_t) {
                                   if (e < M) len[first[i] + e] = x;
                               });
                    const uint32_t m = (uint32_t)kinds[i] >> 4;  // (zeros up to the word's end)
                    if (m + (uint32_t)lane < ((m + 3u) & ~3u)) len[first[i] + m + lane] = 0.0f;
                }
                __syncthreads();
                if (warp == 0 && n == 0) {
                    // One verb of more points than there is room for.
                    const int k = kinds[0] & 15;
                    st.kept += verb_edges(A, S, base, k, P, lane, [&](uint32_t e, uint32_t cnt, float x,
                                                                      uint32_t M, uint32_t m1) {
                        float mine = 0.0f;
                        for (uint32_t j = 0; j < cnt; ++j) {
                            st.adv = st.adv + __shfl_sync(FULL, x, (int)j);
                            if ((uint32_t)lane == j) mine = st.adv;
                        }
                        keep_advancement(out + 4 * (size_t)base, e, M, runs ? m1 : 0u, mine);
                    });
                }
                // The sums of the window's rows of run verbs; lane = verb then takes its four.
                const int mine = warp == 0 && (uint32_t)lane < n ? kinds[lane] : KIND_NONE;
                const uint32_t special = __ballot_sync(FULL, !is_segment(mine & 15));
                for (uint32_t i = 0; warp == 0 && i < n;) {
                    if ((special >> i) & 1u) {
                        advance_special(A, S, base + i, (kinds[i] & 15) & 7, P, st, lane);
                        ++i;
                        continue;
                    }
                    const uint32_t rest = special >> i;
                    const uint32_t end = rest ? min(n, i + (uint32_t)__ffs((int)rest) - 1u) : n;
                    const uint32_t w0 = first[i] / 4u;
                    const uint32_t w1 = (first[end - 1u] + ((uint32_t)kinds[end - 1u] >> 4) + 3u) / 4u;
                    const float start = st.adv;
                    st.adv = running_sums(room + w0, sums + w0, w1 - w0, start, lane);
                    __syncwarp();
                    const float* sum = reinterpret_cast<const float*>(sums);
                    uint32_t m = 0;
                    if ((uint32_t)lane >= i && (uint32_t)lane < end) {
                        m = (uint32_t)mine >> 4;
                        const uint32_t f = first[lane], m1 = split[lane];
                        const float before =
                            (uint32_t)lane == i ? start
                                                : sum[first[lane - 1] +
                                                      ((uint32_t)kinds[lane - 1] >> 4) - 1u];
                        float a[4];
#pragma unroll
                        for (uint32_t c = 0; c < 4; ++c)
                            a[c] = m + c >= 4u ? sum[f + m + c - 4u] : m + c == 3u ? before : 0.0f;
                        if (m1) a[0] = sum[f + m1 - 1u];
                        advancements(S)[base + lane] = make_float4(a[0], a[1], a[2], a[3]);
                    }
                    st.kept += __reduce_add_sync(FULL, m);
                    __syncwarp();
                    i = end;
                }
                base += n > 0 ? n : 1u;
            }
        }
    }
}

// ---- stepping ----------------------------------------------------------------------------------

// One verb's end points, units and how a unit's parameter maps to the curve's (stroke.rs:2755-2779).
struct VerbFeed {
    Unit a, b;
    uint32_t from_id, to_id;
    float sw, ew;  // line widths at its ends
    float ts;      // the parameter of its sharp turn
};
template <bool VW>
__device__ __forceinline__ void load_feed(VerbFeed& f, const StrokeArgs& A, const StrokeVerbs& S,
                                          uint32_t v, float line_width, float tol) {
    const int kind = S.kind[v] & KIND_MASK;
    const uint32_t p = S.rec[v], flags = S.flags[v], cut = flags & VF_TURN ? S.cut[v] : 0u;
    verb_units(kind, p, A.points, tol, flags & VF_TURN, cut, f.a, f.b);
    f.from_id = p - 1;
    f.to_id = p + points_of_verb(kind) - 1;
    f.ts = __uint_as_float(cut);
    if (VW) {
        const size_t ws = A.width_stride ? A.width_stride : 1u;
        f.sw = line_width * A.widths[f.from_id * ws];
        f.ew = line_width * A.widths[f.to_id * ws];
    } else {
        f.sw = f.ew = 0.0f;
    }
}

// Points k0.. of the verb through the stepper; the first one takes the advancement `adv` (NaN: it
// is summed, as the others').
template <bool VW, bool KEEP, class SK>
__device__ __noinline__ void feed_points(Stepper<VW>& stepper, const VerbFeed& feed, bool line,
                                         uint32_t k0, float adv, const StrokeParams& params,
                                         SK& out, int* status, Keep* keep) {
    Stepper<VW> T = stepper;
    SK sink = out;
    const StrokeParams P = params;
    int st = *status;
    const float sw = feed.sw, ew = feed.ew, ts = feed.ts;
    const uint32_t from = feed.from_id, to = feed.to_id, ma = feed.a.m, mb = feed.b.m;
    bool second = mb > 0 && k0 > ma;
    for (;;) {
        const Unit u = second ? feed.b : feed.a;
        uint32_t k = 1;
        if (k0 > 0) k = second ? k0 - ma : k0;
        k0 = 0;
        // The whole curve's parameter: t, or of a split quadratic t * ts and ts + t * (1 - ts).
        const float tmul = mb > 0 ? second ? 1.0f - ts : ts : 1.0f;
        const float tadd = second ? ts : 0.0f;
        float t = k > 1 ? unit_t(u, k - 1u) : 0.0f;
        for (; k <= u.m; ++k) {
            V2 q = u.to;
            if (k == u.m) {
                t = 1.0f;
            } else {
                t = t + u.s;
                q = poly_sample(u.p, t);
            }
            const float w = tadd + t * tmul;
            float hw = P.hw;
            if (VW) hw = line ? ew * 0.5f : (sw * (1.0f - w) + ew * w) * 0.5f;
            stepper_step<VW, KEEP>(T, q, hw, !line && t != 1.0f, adv,
                                   line ? endpoint_src(to) : curve_src(from, to, w), P, sink, st,
                                   keep);
            adv = __int_as_float(0x7fc00000);
        }
        if (second || mb == 0) break;
        second = true;
    }
    stepper = T;
    out = sink;
    *status = st;
}

template <bool VW, bool KEEP, class SK>
__device__ __forceinline__ void feed_begin(Stepper<VW>& T, const StrokeArgs& A,
                                           const StrokeVerbs& S, uint32_t v, float line_width,
                                           const StrokeParams& P, float adv, SK& sink,
                                           int* status, Keep* keep) {
    const uint32_t p = S.rec[v];
    const size_t ws = A.width_stride ? A.width_stride : 1u;
    stepper_step<VW, KEEP>(T, load_pt(A.points, p),
                           VW ? line_width * A.widths[p * ws] * 0.5f : P.hw, false, adv,
                           endpoint_src(p), P, sink, *status, keep);
}

// Steps the last kept points before the verb in slot `v`: at least four, or all from the
// sub-path's Begin. Goes back over six verbs at most: each keeps a point at least, and of two in a
// row the end point of one at least (drops_kernel), from which the steps can start when four points
// follow it.
template <bool VW, bool KEEP, class SK>
__device__ __noinline__ void warm_up(Stepper<VW>& St, const StrokeArgs& A, const StrokeVerbs& S,
                                     uint32_t v, float lw, const StrokeParams& P, SK& sink,
                                     int* status, Keep* keep) {
    constexpr bool ADV = VW || SK::kRec;
    uint32_t u = v - 1, have = 0, k0 = 0;  // k0 == 0: from the Begin in u
    for (;;) {
        const int kind = S.kind[u] & KIND_MASK;
        if (kind == LYON_VERB_BEGIN) break;
        const uint32_t f = S.flags[u], nk = flags_nk(f);
        // Of a verb whose steps are all kept the last ones are enough, unless a cusp is near
        // (its sides hang on the points before it).
        const bool end = have >= 4u && !(f & VF_MERGED);
        const uint32_t need = have >= 4u ? 1u : 4u - have;
        if (end || (!(f & VF_IRR) && (nk >= need || nk >= 3u))) {
            VerbFeed x;
            load_feed<VW>(x, A, S, u, lw, P.tolerance);
            const uint32_t all = x.a.m + x.b.m, cut = f & VF_CUT ? S.cut[u] : 0u;
            if (end || (all >= need && cut <= 0xFFFFu && (cut == 0 || all - cut >= 8u))) {
                k0 = all - need + 1u;
                feed_points<VW, KEEP>(St, x, kind == LYON_VERB_LINE_TO, k0,
                                      ADV ? advancement_back(S, u, need - 1u)
                                          : __int_as_float(0x7fc00000),
                                      P, sink, status, keep);
                break;
            }
        }
        have += nk;
        --u;
    }
    if (k0 == 0)
        feed_begin<VW, KEEP>(St, A, S, u, lw, P, ADV ? advancement_back(S, u, 0) : 0.0f, sink,
                             status, keep);
    for (++u; u < v; ++u) {
        VerbFeed x;
        load_feed<VW>(x, A, S, u, lw, P.tolerance);
        feed_points<VW, KEEP>(St, x, (S.kind[u] & KIND_MASK) == LYON_VERB_LINE_TO, 1u,
                              __int_as_float(0x7fc00000), P, sink, status, keep);
    }
}

// What the stepper's next steps read of its state; ids count back from the next one.
__device__ __forceinline__ unsigned long long mix(unsigned long long h, uint32_t x) {
    h = (h ^ x) * 0x9E3779B97F4A7C15ull;
    return h ^ (h >> 29);
}
template <bool VW>
__device__ __forceinline__ unsigned long long state_hash(const Stepper<VW>& T, uint32_t next_id) {
    unsigned long long h = mix(0x243F6A8885A308D3ull, T.count * 4u + (T.lflat ? 1u : 0u));
    const float v[] = {T.ppos.x, T.ppos.y, T.pnext_p.x, T.pnext_p.y, T.pnext_n.x, T.pnext_n.y,
                       T.padv, T.phw, T.lpos.x, T.lpos.y, T.lprev_p.x, T.lprev_p.y, T.lprev_n.x,
                       T.lprev_n.y, T.ladv, T.lhw};
#pragma unroll
    for (int i = 0; i < 16; ++i) h = mix(h, isnan(v[i]) ? 1u : __float_as_uint(v[i]));
    h = mix(h, T.pneg == INVALID_ID ? INVALID_ID : next_id - T.pneg);
    return mix(h, T.ppid == INVALID_ID ? INVALID_ID : next_id - T.ppid);
}

// (Ids counted from `id_base`: only whether two are equal matters without output.)
template <class SK>
__device__ __forceinline__ void silent_sink(SK& s, uint32_t id_base) {
    s.id_base = id_base;
    s.nv = s.ni = 0;
    s.vout = nullptr;
    s.rout = nullptr;
    s.iout = nullptr;
    s.index_bits = 32;
    s.vcap = s.icap = 0;
    s.overflow = false;
    s.adv = 0.0f;
    set_sout(s, nullptr);
    set_src(s, endpoint_src(LYON_NO_ENDPOINT));
}
// Turns the sink that warmed up into one that writes at (vo, io) of the path, ids with it.
template <bool VW, class SK>
__device__ __forceinline__ void aim_sink(Stepper<VW>& T, Keep* keep, SK& s, const StrokeArgs& A,
                                         uint32_t path, const PathOut& po, uint32_t vo,
                                         uint32_t io) {
    const uint32_t shift = po.id_base + vo - (s.id_base + s.nv);
    if (T.pneg != INVALID_ID) T.pneg += shift;
    if (T.ppid != INVALID_ID) T.ppid += shift;
    if (keep) {
        for (int k = 0; k < 2; ++k) {
            SidePts& q = keep->join.s[k];
            if (q.prev_vertex != INVALID_ID) q.prev_vertex += shift;
            if (q.next_vertex != INVALID_ID) q.next_vertex += shift;
        }
    }
    s.id_base = po.id_base + vo;
    s.nv = s.ni = 0;
    s.vout = po.vout ? po.vout + vo : nullptr;
    s.rout = po.rout ? po.rout + vo : nullptr;
    s.iout = po.bits == 16 ? (void*)((uint16_t*)po.iout + io) : (void*)((uint32_t*)po.iout + io);
    s.index_bits = po.bits;
    s.vcap = cap_left(po.vmax, vo);
    s.icap = cap_left(po.imax, io);
    s.overflow = false;
    set_sout(s, A.sources + A.vtx_offsets[path] + vo);
}

// Where the output of the segment in slot `v` starts and ends when it begins with the join at the
// verb before's last point, from the counts of stroke_verbs.cu (which give that join to that verb).
struct Span {
    uint32_t v0, i0, v1, i1;
};
__device__ __forceinline__ void end_join_size(const StrokeVerbs& S, uint32_t v, uint32_t* nv,
                                              uint32_t* ni) {
    const uint32_t join = S.join[v], flags = S.flags[v];
    uint32_t edge = 0;
    if (flags_nk(flags) >= 2) {
        const bool own = (flags & VF_IRR) || ((flags & VF_TWO) && (flags & VF_SECOND1));
        edge = edge_count_flags(pj_from(own ? S.split[v] : PACKED_STEP), pj_to(join));
    } else if ((S.kind[v - 1] & KIND_MASK) != LYON_VERB_BEGIN) {
        edge = edge_count_flags(pj_from(S.join[v - 1]), pj_to(join));
    }
    *nv = pj_vertices(join);
    *ni = 3u * (edge + pj_tris(join));
}
template <bool VW>
__device__ __forceinline__ Span verb_span(const StrokeVerbs& S, uint32_t v, uint32_t path) {
    Span r{S.vpre[v] - S.path_v[path], S.ipre[v] - S.path_i[path],
           S.vpre[v + 1] - S.path_v[path], S.ipre[v + 1] - S.path_i[path]};
    if (!VW && is_segment(S.kind[v] & KIND_MASK)) {
        uint32_t a, b;
        if ((S.kind[v - 1] & KIND_MASK) != LYON_VERB_BEGIN) {
            end_join_size(S, v - 1, &a, &b);
            r.v0 -= a;
            r.i0 -= b;
        }
        if (is_segment(S.kind[v + 1] & KIND_MASK)) {
            end_join_size(S, v, &a, &b);
            r.v1 -= a;
            r.i1 -= b;
        }
    }
    return r;
}

// One verb: its points through the stepper, or the end of its sub-path.
template <bool EMIT, bool VW, class SK>
__device__ __forceinline__ void step_verb(const StrokeArgs& A, const StrokeVerbs& S, uint32_t v) {
    const uint32_t path = S.path[v];
    if (S.path_walk[path] || (EMIT && A.status[path] != LYON_OK)) return;
    const lyon_stroke_options opt = A.options[A.num_options > 1 ? path : 0];
    const StrokeParams P = make_params(opt);
    const int kind = S.kind[v] & KIND_MASK;
    PathOut po = path_out<EMIT, SK::kRec>(A, path);
    Span sp{0, 0, 0, 0};
    if (EMIT) sp = verb_span<VW>(S, v, path);
    Stepper<VW> T;
    stepper_init(T);
    SK s;
    silent_sink(s, 1u << 28);
    int status = LYON_OK;
    uint32_t nv0 = 0, ni0 = 0;
    if (is_segment(kind)) {
        warm_up<VW, false>(T, A, S, v, opt.line_width, P, s, &status, nullptr);
        if (EMIT) {
            aim_sink<VW>(T, nullptr, s, A, path, po, sp.v0, sp.i0);
        } else {
            nv0 = s.nv;
            ni0 = s.ni;
            if (VW) state_hashes(S)[v].x = state_hash(T, s.id_base + s.nv);
        }
        VerbFeed x;
        load_feed<VW>(x, A, S, v, opt.line_width, P.tolerance);
        feed_points<VW, false>(T, x, kind == LYON_VERB_LINE_TO, 1u, __int_as_float(0x7fc00000), P,
                               s, &status, nullptr);
        if (!EMIT && VW) state_hashes(S)[v].y = state_hash(T, s.id_base + s.nv);
    } else {
        // The first two points with their sides and ids (lyon's firsts): the sub-path's first
        // steps, as they were when its first join's vertices were written.
        constexpr bool ADV = VW || SK::kRec;
        const uint32_t b = S.rec[v];
        Keep keep;
        keep.nfirsts = 0;
        keep.mnec = false;
        if (EMIT) s.id_base = po.id_base + S.vpre[b] - S.path_v[path];
        feed_begin<VW, true>(T, A, S, b, opt.line_width, P, ADV ? advancement_back(S, b, 0) : 0.0f,
                             s, &status, &keep);
        uint32_t u = b + 1;
        for (; u < v && keep.nfirsts < 2; ++u) {
            VerbFeed x;
            load_feed<VW>(x, A, S, u, opt.line_width, P.tolerance);
            feed_points<VW, true>(T, x, (S.kind[u] & KIND_MASK) == LYON_VERB_LINE_TO, 1u,
                                  __int_as_float(0x7fc00000), P, s, &status, &keep);
        }
        if (u < v) {
            // More points follow: the state at the end, with the firsts of the beginning.
            const DEP f0 = keep.first[0], f1 = keep.first[1];
            const lyon_vertex_source s0 = keep.first_src;
            stepper_init(T);
            silent_sink(s, 1u << 29);
            warm_up<VW, true>(T, A, S, v, opt.line_width, P, s, &status, &keep);
            keep.first[0] = f0;
            keep.first[1] = f1;
            keep.first_src = s0;
            keep.nfirsts = 2;
        }
        keep.mnec = (S.kind[v] & KIND_MNEC) != 0;
        if (EMIT) {
            aim_sink<VW>(T, &keep, s, A, path, po, sp.v0, sp.i0);
        } else {
            nv0 = s.nv;
            ni0 = s.ni;
            if (VW) state_hashes(S)[v].x = state_hash(T, s.id_base + s.nv);
        }
        float start_adv = ADV ? advancement_back(S, b, 0) : 0.0f;
        stepper_end<VW>(T, keep, kind == LYON_VERB_CLOSE, P, s, &status, &start_adv);
        // Where the path's next sub-path starts, against what advance_special took: a skipped step
        // replaces a point of a variable-width stroke, and the sum over its points is another one.
        // (Not only records show it: a join's fold test takes differences of advancements, which
        // round by their size.)
        if (VW && !EMIT && v + 1u < A.verb_offsets[path + 1] - A.verb_offsets[0] &&
            (S.kind[v + 1] & KIND_MASK) == LYON_VERB_BEGIN &&
            !(start_adv == advancement_back(S, v + 1, 0)))
            leave_to_walk(S, path);
    }
    if (EMIT) {
        if (s.overflow && status == LYON_OK) status = LYON_ERR_INTERNAL;
        if (status != LYON_OK || sp.v0 + s.nv != sp.v1 || sp.i0 + s.ni != sp.i1)
            A.status[path] = status != LYON_OK ? status : LYON_ERR_INTERNAL;
    } else {
        if (status != LYON_OK) leave_to_walk(S, path);
        S.vpre[v] = s.nv - nv0;
        S.ipre[v] = s.ni - ni0;
    }
}

// Threads take the verbs of a tile sorted by what they are (curves, lines, ends; each from a warp's
// boundary), so that the lanes of a warp do much the same. In full tiles the kinds follow one another,
// so that a block's warps share their instructions (10,001 curve paths of variable width 6.8 ms, with
// the kinds side by side 7.1). A batch too small for a full tile per block has smaller tiles, with
// the kinds side by side: 100 lines of four points and variable width 343 -> 173 us.
constexpr uint32_t STEP_TILE = 512, STEP_TILE_LEAST = 32;
template <bool EMIT, bool VW, class SK>
__global__ void __launch_bounds__(128) steps_kernel(StrokeArgs A, StrokeVerbs S) {
    __shared__ uint16_t list[3][STEP_TILE];
    __shared__ uint32_t count[3];
    const uint32_t nv = batch_verbs(A);
    if (unfit(S, nv)) return;
    const uint32_t size = tile_size(nv, STEP_TILE_LEAST, STEP_TILE);
    for (uint32_t tile = blockIdx.x * size; tile < nv; tile += gridDim.x * size) {
        __syncthreads();
        if (threadIdx.x < 3) count[threadIdx.x] = 0;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < size && tile + i < nv; i += blockDim.x) {
            const int k = S.kind[tile + i] & KIND_MASK;
            const int l = k == LYON_VERB_LINE_TO ? 1 : is_segment(k) ? 0 : is_end(k) ? 2 : 3;
            if (l < 3) list[l][atomicAdd(&count[l], 1u)] = (uint16_t)i;
        }
        __syncthreads();
        const uint32_t n0 = count[0], n1 = count[1], n2 = count[2];
        const uint32_t s1 = (n0 + 31u) & ~31u, s2 = s1 + ((n1 + 31u) & ~31u);
        const bool apart = size == STEP_TILE;
        for (int pass = 0; pass < (apart ? 3 : 1); ++pass) {
            const uint32_t from = pass == 0 ? 0u : pass == 1 ? s1 : s2;
            const uint32_t to = !apart || pass == 2 ? s2 + n2 : pass == 0 ? s1 : s2;
            for (uint32_t i = from + threadIdx.x; i < to; i += blockDim.x) {
                const int l = i < s1 ? 0 : i < s2 ? 1 : 2;
                const uint32_t j = l == 0 ? i : l == 1 ? i - s1 : i - s2;
                if (j < (l == 0 ? n0 : l == 1 ? n1 : n2))
                    step_verb<EMIT, VW, SK>(A, S, tile + list[l][j]);
            }
            if (apart) __syncthreads();
        }
    }
}

// Every verb's state against the one the verb before left.
__global__ void __launch_bounds__(256) check_states_kernel(StrokeArgs A, StrokeVerbs S) {
    const uint32_t nv = batch_verbs(A);
    if (unfit(S, nv)) return;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nv;
         v += gridDim.x * blockDim.x) {
        const int kind = S.kind[v] & KIND_MASK;
        if (!is_segment(kind) && !is_end(kind)) continue;
        if (S.path_walk[S.path[v]] || !is_segment(S.kind[v - 1] & KIND_MASK)) continue;
        if (state_hashes(S)[v].x != state_hashes(S)[v - 1].y) leave_to_walk(S, S.path[v]);
    }
}

uint32_t blocks_for(uint32_t items, uint32_t per_block, int num_sms, uint32_t waves) {
    const uint32_t sms = (uint32_t)(num_sms > 0 ? num_sms : 1);
    const uint32_t need = (items + per_block - 1) / per_block;
    return need < sms ? sms : need > sms * waves ? sms * waves : need;
}

}  // namespace

// On two side streams, which the caller joins: the long paths are few blocks, each bound by its chain
// of additions (20,000 paths with records: 0.74 and 0.62 ms one after the other). They read what
// drops_kernel leaves.
void launch_stroke_advance(const StrokeArgs& a, const StrokeVerbs& v, int num_sms,
                           const SideStreams& side, cudaStream_t s) {
    const cudaStream_t w = side.fork(1, s), l = side.fork(2, s);
    advance_long_kernel<<<blocks_for(a.num_paths, 1, num_sms, 8), 256, 0, l>>>(a, v);
    advance_kernel<<<blocks_for(a.num_paths, 4, num_sms, 16), 128, 0, w>>>(a, v);
    note_launches(2);
}
void join_stroke_advance(const SideStreams& side, cudaStream_t s) {
    side.join(1, s);
    side.join(2, s);
}

void launch_stroke_steps_count(const StrokeArgs& a, const StrokeVerbs& v, uint32_t verbs_hint,
                               int num_sms, const SideStreams& side, cudaStream_t s) {
    launch_stroke_advance(a, v, num_sms, side, s);
    join_stroke_advance(side, s);
    steps_kernel<false, true, Sink>
        <<<blocks_for(verbs_hint, STEP_TILE, num_sms, 16), 128, 0, s>>>(a, v);
    check_states_kernel<<<blocks_for(verbs_hint, 256, num_sms, 8), 256, 0, s>>>(a, v);
    note_launches(2);
}

cudaError_t launch_stroke_steps_emit(const StrokeArgs& a, const StrokeVerbs& v,
                                     uint32_t verbs_hint, int num_sms, const SideStreams& side,
                                     cudaStream_t s) {
    const uint32_t grid = blocks_for(verbs_hint, STEP_TILE, num_sms, 16);
    if (a.widths) {
        if (a.sources && a.vertex_attrs) {
            steps_kernel<true, true, SrcSinkT<true>><<<grid, 128, 0, s>>>(a, v);
        } else if (a.sources) {
            steps_kernel<true, true, SrcSinkT<false>><<<grid, 128, 0, s>>>(a, v);
        } else if (a.vertex_attrs) {
            steps_kernel<true, true, RecSink><<<grid, 128, 0, s>>>(a, v);
        } else {
            steps_kernel<true, true, Sink><<<grid, 128, 0, s>>>(a, v);
        }
    } else {
        if (a.vertex_attrs) {
            if (a.num_paths > STROKE_ADVANCE_EARLY) {
                launch_stroke_advance(a, v, num_sms, side, s);
                join_stroke_advance(side, s);
            }
            steps_kernel<true, false, SrcSinkT<true>><<<grid, 128, 0, s>>>(a, v);
        } else {
            steps_kernel<true, false, SrcSinkT<false>><<<grid, 128, 0, s>>>(a, v);
        }
    }
    note_launches(1);
    return cudaGetLastError();
}

}  // namespace lg
