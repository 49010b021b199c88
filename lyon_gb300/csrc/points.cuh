// points.cuh — the flattened points of many curves at once, lane = point.
#pragma once

#include "geom.cuh"

namespace lg {
namespace {

constexpr uint32_t FULL = 0xFFFFFFFFu;

// A flattened curve, or part of one.
struct Unit {
    Poly p;
    V2 to;
    float s, t0;  // lyon's step 1/n and the parameter the unit starts from
    uint32_t m;   // steps (the last one is `to`); 0: no such unit
};

__device__ __forceinline__ void unit_of(Unit& u, const Poly& p, V2 to, float n) {
    u.p = p;
    u.to = to;
    u.s = 1.0f / n;
    u.t0 = 0.0f;
    u.m = to_u32_or1(n);
}
__device__ __forceinline__ float unit_t(const Unit& u, uint32_t k) {
    return accumulate_t(u.s, 0, u.t0, k);
}

// ---- windows of points -------------------------------------------------------------------------
// A warp takes a window of verbs and works on all points of their units, 32 at a time, lane =
// point, whatever the units' lengths. Point k of a unit (1 to m; point m is its end) has lyon's
// t_k = t_(k-1) + 1/n.
constexpr int WIN_WARPS = 4;
constexpr uint32_t WIN_VERBS = 32;            // verbs per window
constexpr uint32_t WIN_UNITS = 2 * WIN_VERBS;
constexpr uint32_t WIN_ROUND = 512;           // points laid out at a time
struct PointSmem {
    float t[WIN_ROUND];
    uint8_t owner[WIN_ROUND];
};
// A unit as the points read it: four 16-byte words.
struct __align__(16) UnitSmem {
    float4 a01, a23;     // the polynomial
    float4 c1_to;        // the kept point before the unit, its end point
    float s, t0;
    uint32_t m_cubic;    // steps, times two; bit 0: the polynomial is cubic
    uint32_t excl;       // its first point within the window's points
};
__device__ __forceinline__ void lay_out_unit(UnitSmem& r, const Unit& u, V2 from, uint32_t first) {
    r.a01 = make_float4(u.p.a0.x, u.p.a0.y, u.p.a1.x, u.p.a1.y);
    r.a23 = make_float4(u.p.a2.x, u.p.a2.y, u.p.a3.x, u.p.a3.y);
    r.c1_to = make_float4(from.x, from.y, u.to.x, u.to.y);
    r.s = u.s;
    r.t0 = u.t0;
    r.m_cubic = 2u * u.m + (u.p.cubic ? 1u : 0u);
    r.excl = first;
}
// Lays out points [r0, r0 + rn) of the units: a lane takes WIN_ROUND / 32 points in a row, jumps to
// the t before its first one and adds the step from there.
__device__ __forceinline__ void fill_points(PointSmem& sm, const UnitSmem* units, size_t stride,
                                            uint32_t nunits, uint32_t r0, uint32_t rn, int lane) {
    auto unit = [&](uint32_t u) -> const UnitSmem& {
        return *reinterpret_cast<const UnitSmem*>(reinterpret_cast<const char*>(units) + u * stride);
    };
    constexpr uint32_t PER = WIN_ROUND / 32;
    uint32_t i = (uint32_t)lane * PER;
    if (i < rn) {
        uint32_t lo = 0, hi = nunits - 1;  // the last unit that starts at or before the point
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1) >> 1;
            if (unit(mid).excl <= r0 + i) lo = mid; else hi = mid - 1;
        }
        const uint32_t end = min(i + PER, rn);
        uint32_t u = lo, k = r0 + i - unit(u).excl, m = unit(u).m_cubic >> 1;
        float s = unit(u).s, t = accumulate_t(s, 0, unit(u).t0, k);
        for (; i < end; ++i) {
            if (k == m) {
                ++u;
                k = 0;
                m = unit(u).m_cubic >> 1;
                s = unit(u).s;
                t = unit(u).t0;
            }
            t = t + s;
            sm.t[i] = t;
            sm.owner[i] = (uint8_t)u;
            ++k;
        }
    }
    __syncwarp();
}
// Point k of a unit at t (poly_sample's operations).
__device__ __forceinline__ V2 unit_point(const UnitSmem& r, uint32_t k, float t) {
    const float4 p = r.a01, q = r.a23, e = r.c1_to;
    const float t2 = t * t, t3 = t2 * t;
    float x = (p.x + p.z * t) + q.x * t2, y = (p.y + p.w * t) + q.y * t2;
    const float x3 = x + q.z * t3, y3 = y + q.w * t3;
    const bool cubic = (r.m_cubic & 1u) != 0, end = k == (r.m_cubic >> 1);
    x = cubic ? x3 : x;
    y = cubic ? y3 : y;
    return V2{end ? e.z : x, end ? e.w : y};
}
// The value of the lane before; lane 0 takes lane 31's of the chunk before (`old`).
__device__ __forceinline__ float from_left(float now, float old, int lane) {
    return __shfl_sync(FULL, lane == 31 ? old : now, (lane + 31) & 31);
}
// Verbs per window: fewer in a small batch, so that every warp of the grid has a window.
__device__ __forceinline__ uint32_t window_verbs(uint32_t nv, uint32_t nwarps) {
    return max(1u, min(WIN_VERBS, nv / (2u * nwarps)));
}

}  // namespace
}  // namespace lg
