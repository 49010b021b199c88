// flatten.cu — path flattening: per-verb segment counts and `path.iter().flattened(tol)`.
//
// Counts: one warp per path, verbs in windows of 32 (lane = verb): a warp scan of the points per
// verb gives each verb its points, lyon's `flattened_segments_wang` gives each curve its segment
// count (crates/geom/src/quadratic_bezier.rs:943-974, crates/geom/src/cubic_bezier.rs:1369-1403).
// Points: windows of 32 verbs of the whole batch, lane = flattened point: lyon's Horner polynomial
// at the accumulated parameter (crates/geom/src/quadratic_bezier.rs:1004-1033 and
// crates/geom/src/cubic_bezier.rs:1434-1459 iterators). A point's neighbour in memory is its
// neighbour in the warp, across verbs and paths.
#include "points.cuh"
#include "kernels.h"
#include "kernels_flatten.h"

namespace lg {

__device__ __forceinline__ uint32_t fl_points_of_verb(int kind) {
    switch (kind) {
        case LYON_VERB_LINE_TO: return 1;
        case LYON_VERB_QUADRATIC_TO: return 2;
        case LYON_VERB_CUBIC_TO: return 3;
        case LYON_VERB_BEGIN: return 1;
        case LYON_VERB_CLOSE: return 1;
        default: return 0;
    }
}

// The flattened curve of a verb whose points start at `p`; m == 0: it contributes no points.
__device__ __forceinline__ Unit verb_unit(int kind, uint32_t p, const float* points, float tol) {
    Unit u;
    u.m = 0;
    u.s = 1.0f;
    u.t0 = 0.0f;
    if (kind == LYON_VERB_LINE_TO) {
        u.p = Poly{V2{0.0f, 0.0f}, V2{0.0f, 0.0f}, V2{0.0f, 0.0f}, V2{0.0f, 0.0f}, false};
        u.to = load_pt(points, p);
        u.m = 1;
    } else if (kind == LYON_VERB_QUADRATIC_TO) {
        const V2 from = load_pt(points, p - 1), c = load_pt(points, p), to = load_pt(points, p + 1);
        unit_of(u, quad_poly(from, c, to), to, quad_wang(from, c, to, tol));
    } else if (kind == LYON_VERB_CUBIC_TO) {
        const V2 from = load_pt(points, p - 1), c1 = load_pt(points, p);
        const V2 c2 = load_pt(points, p + 1), to = load_pt(points, p + 2);
        unit_of(u, cubic_poly(from, c1, c2, to), to, cubic_wang(from, c1, c2, to, tol));
    }
    return u;
}

// Counts per verb, and (`firsts`, optional) where a counted verb's points start.
__global__ void __launch_bounds__(256) flatten_count_kernel(FlattenArgs A) {
    const int lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    // (The arrays end with the last path's verbs, also where offsets run backwards.)
    const uint32_t v_last = A.verb_offsets[A.num_paths];
    for (uint32_t path = warp; path < A.num_paths; path += nwarps) {
        const uint32_t v_begin = A.verb_offsets[path];
        const uint32_t v_end = min(A.verb_offsets[path + 1], v_last);
        uint32_t pc = A.point_offsets[path];
        const uint32_t p_end = A.point_offsets[path + 1];
        for (uint32_t vi = v_begin; vi < v_end; vi += 32) {
            const uint32_t v = vi + (uint32_t)lane;
            const bool valid = v < v_end;
            const int kind = valid ? (int)A.verbs[v] : LYON_VERB_END;
            const uint32_t pcount = valid ? fl_points_of_verb(kind) : 0u;
            uint32_t incl = pcount;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t up = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += up;
            }
            const uint32_t pofs = pc + incl - pcount;
            const bool ok = valid && pofs + pcount <= p_end && pofs >= 1;
            const uint32_t n = ok ? verb_unit(kind, pofs, A.points, A.tolerance).m : 0u;
            if (valid) {
                A.counts[v] = n;
                if (A.firsts) A.firsts[v] = n > 0 ? pofs : FLATTEN_NO_POINTS;
            }
            pc += __shfl_sync(FULL, incl, 31);
        }
    }
}

constexpr uint32_t FLATTEN_BIG = 1u << 20;

struct FlatSlot {
    UnitSmem u;
    float2* out;
    uint32_t pad[2];
};
struct FlatSmem {
    FlatSlot unit[WIN_VERBS];
    PointSmem pt;
};

// Bound by instruction issue (about 60 per 32 points) and the stores, 8 bytes a lane in a row.
// Measured on 40,000 curve paths at tolerance 0.02 (the whole call, the points copied on): 0.64 ms
// (this kernel 0.35); 4.58 ms with one warp per path, which found each point's verb by bisection
// over shuffles and its parameter from the curve's start.
__global__ void __launch_bounds__(WIN_WARPS * 32) flatten_points_kernel(FlattenArgs A, uint32_t nv) {
    __shared__ FlatSmem smem[WIN_WARPS];
    const int lane = threadIdx.x & 31;
    FlatSmem& sm = smem[threadIdx.x >> 5];
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t W = window_verbs(nv, nwarps);
    for (uint32_t w0 = warp * W; w0 < nv; w0 += nwarps * W) {
        const uint32_t v = w0 + (uint32_t)lane;
        Unit u;
        u.m = 0;
        if ((uint32_t)lane < W && v < nv) {
            const uint32_t p = A.firsts[v];
            if (p != FLATTEN_NO_POINTS) u = verb_unit(A.verbs[v], p, A.points, A.tolerance);
        }
        // Curves of very many points, one after the other (sums of their counts would overflow).
        uint32_t big = __ballot_sync(FULL, u.m > FLATTEN_BIG);
        while (big) {
            const uint32_t bv = w0 + (uint32_t)__ffs(big) - 1u;
            big &= big - 1u;
            const Unit x = verb_unit(A.verbs[bv], A.firsts[bv], A.points, A.tolerance);
            float2* out = reinterpret_cast<float2*>(A.out_points) + A.offsets[bv];
            for (uint64_t k = (uint64_t)lane + 1u; k <= x.m; k += 32) {
                const V2 q = k == x.m ? x.to : poly_sample(x.p, unit_t(x, (uint32_t)k));
                out[k - 1u] = make_float2(q.x, q.y);
            }
        }
        if (u.m > FLATTEN_BIG) u.m = 0;
        const uint32_t mask = __ballot_sync(FULL, u.m > 0);
        if (mask == 0) continue;
        uint32_t incl = u.m;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t up = __shfl_up_sync(FULL, incl, d);
            if (lane >= d) incl += up;
        }
        const uint32_t total = __shfl_sync(FULL, incl, 31);
        if (u.m > 0) {
            FlatSlot& r = sm.unit[__popc(mask & ((1u << lane) - 1u))];
            lay_out_unit(r.u, u, u.to, incl - u.m);
            r.out = reinterpret_cast<float2*>(A.out_points) + A.offsets[v];
        }
        __syncwarp();
        for (uint32_t r0 = 0; r0 < total; r0 += WIN_ROUND) {
            const uint32_t rn = min(WIN_ROUND, total - r0);
            fill_points(sm.pt, &sm.unit[0].u, sizeof(FlatSlot), (uint32_t)__popc(mask), r0, rn, lane);
            for (uint32_t i = (uint32_t)lane; i < rn; i += 32) {
                const FlatSlot& r = sm.unit[sm.pt.owner[i]];
                const uint32_t k = r0 + i - r.u.excl + 1u;
                const V2 q = unit_point(r.u, k, sm.pt.t[i]);
                r.out[k - 1u] = make_float2(q.x, q.y);
            }
            __syncwarp();
        }
    }
}

cudaError_t launch_flatten_counts(const FlattenArgs& a, int num_sms, cudaStream_t s) {
    flatten_count_kernel<<<num_sms * 8, 256, 0, s>>>(a);
    note_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_flatten_points(const FlattenArgs& a, uint32_t num_verbs, int num_sms,
                                  cudaStream_t s) {
    if (num_verbs == 0) return cudaSuccess;
    flatten_points_kernel<<<num_sms * 8, WIN_WARPS * 32, 0, s>>>(a, num_verbs);
    note_launches(1);
    return cudaGetLastError();
}

}  // namespace lg
