// fill_warp.cuh — lyon's FillTessellator run by one warp per path (see fill.cu for the batching).
//
// The sweep line is sequential within a path: every event depends on the active edges that the
// event before it left. What one event does is wide, though, and a path's other steps are not
// sequential at all, so a warp works on one path:
//   * event queue: the points of a curve are flattened one per lane, their edges and vertex events
//     packed by ballots in lyon's order; the events are ordered by a stable merge sort whose
//     elements find their places by binary search, and copied in that order, so that the sweep
//     reads them one after another and has the next one loaded before it needs it;
//   * an event: each lane holds one active edge of the current 32; the scan, the check of the
//     remaining edges and the intersection tests are a few ballots, the winding in front of the
//     point is a population count. All lanes run the scalar steps between with the same values;
//   * monotone tessellators: the sweep only appends (vertex, side) to the spans' vertex lists. The
//     spans are independent of one another once their lists are known, so after the last event
//     each lane triangulates one span. A span of k vertices that is ended gives k - 2 triangles,
//     which places its output; spans are written in the order in which lyon flushes them.
// The active edges, pending edges and span list of a path are in shared memory as long as they
// fit (longer ones move to the heap).
//
// What bounds it: the dependent instructions of one event after another (about 700 instructions, 7
// cycles each with four warps on an SM; 40 % of that is fixed latency). Code size comes next: with 16
// warps on an SM, each at another place of 250 KB of code, a warp waited for its next instruction
// 60 % of the time, so rare steps are out of line and loops are not unrolled (143 KB: 30,000 glyph
// paths 1.5 times faster). Times, a thread per path and a warp per path: one glyph of 1,083 events
// 11.6 and 2.9 ms, 777 glyphs 47.8 and 9.8 ms, 30,000 glyphs 361 and 53 ms. Small simple paths of large
// batches are the thread's (fill.cu has the rule and both sides' figures).
// Warps per SM, for one glyph / 777 / 30,000: 8 (154 registers) 2.8 / 9.6 / 68 ms, 12 2.9 / 9.6 / 59,
// 16 (128 registers) 3.0 / 10.0 / 55, 20 3.1 / 10.4 / 53, 24 3.3 / 10.6 / 54, 32 3.8 / 11.3 / 58.
#pragma once

#include "fill_core.cuh"

namespace lg {
namespace fillk {

constexpr uint32_t FULL = 0xFFFFFFFFu;
constexpr uint32_t SMEM_ACTIVE = 64, SMEM_BELOW = 8, SMEM_SPANS = 32;

// The warp's piece of device memory, handed out upwards in 16-byte steps. The arrays that building
// the event queue needs are dead once the events are in order: [lo, lo_end) is their room, used
// again before the rest.
struct WarpHeap {
    uint32_t* w;
    uint32_t cap, top;
    uint32_t lo, lo_end;
};

// ---- sweep structures (fill.rs) --------------------------------------------------------------

// fill.rs:185-200 with geom line.rs:56-71
__device__ __forceinline__ float min_x(V2 from, V2 to) { return fminf(from.x, to.x); }
__device__ __forceinline__ float max_x(V2 from, V2 to) { return from.x > to.x ? from.x : to.x; }
__device__ __forceinline__ float solve_x_for_y(V2 from, V2 to, float y) {
    float dy = to.y - from.y;
    float t = dy == 0.0f ? 0.0f : (y - from.y) / dy;
    float x = from.x * (1.0f - t) + to.x * t;
    return fminf(fmaxf(x, min_x(from, to)), max_x(from, to));
}

// An active edge (fill.rs:153-170) is two 16-byte words: from and to; then the winding (its low
// 16 bits, with AE_MERGE above them), the id of `from`, the source edge's event and range_end.
constexpr uint32_t AE_MERGE = 1u << 16;
__device__ __forceinline__ V2 ae_from(float4 a) { return V2{a.x, a.y}; }
__device__ __forceinline__ V2 ae_to(float4 a) { return V2{a.z, a.w}; }
__device__ __forceinline__ bool ae_is_merge(uint4 b) { return (b.x & AE_MERGE) != 0; }
__device__ __forceinline__ int32_t ae_winding(uint4 b) { return (int32_t)(int16_t)(b.x & 0xFFFFu); }

struct __align__(16) WarpPending {  // fill.rs:304-312
    V2 to;
    float sort_key, range_end;
    uint32_t src_edge;
    int32_t winding;
    uint32_t pad[2];
};

// The first test of segment_intersection_t (geom line.rs:217-253): a shared end point.
__device__ __forceinline__ bool share_end_point(V2 sf, V2 st, V2 of, V2 ot) {
    return peq(st, ot) || peq(sf, of) || peq(sf, ot) || peq(st, of);
}
// segment_intersection_t, once in the instruction cache.
__device__ __noinline__ bool intersection_t(V2 sf, V2 st, V2 of, V2 ot, double* ta, double* tb) {
    return segment_intersection_t(sf.x, sf.y, st.x, st.y, of.x, of.y, ot.x, ot.y, ta, tb);
}

// The event queue (event_queue.rs): one entry per event in each array. `wind` holds the winding in
// its low 16 bits and IS_EDGE above them; `link` the next sibling and the next event; `ids`, with
// sources only, the path-local endpoint ids of the event's source edge.
constexpr uint32_t IS_EDGE = 1u << 16;
struct Events {
    V2* pos;
    float4* edge;  // to, range_start, range_end
    uint32_t* wind;
    uint2* link;
    uint2* ids;
    uint32_t n, cap;
};

// What a warp keeps in shared memory.
struct __align__(16) SweepSmem {
    float4 act_a[SMEM_ACTIVE];
    uint4 act_b[SMEM_ACTIVE];
    WarpPending below[SMEM_BELOW];
    uint2 spans[SMEM_SPANS];
    WarpHeap heap;
    Events ev;
    uint32_t sorted_n;  // events [0, sorted_n) are in order of position
    // Output vertices and, with sources, FillVertex::sources (three words each, path-local ids)
    // and each vertex's first source.
    V2* out_v;
    uint32_t* out_src;
    uint32_t* out_sfirst;
    uint32_t out_cap, src_cap, sfirst_cap;
    // Spans by uid: the first vertex (position, id), the list's length and place; the uids in the
    // order of their flushes (bit 31: not ended).
    float4* span_first;
    uint2* span_len;
    uint32_t* flushed;
    uint32_t uid_cap, len_cap, flushed_cap;
    // The (uid, vertex | side << 31) and the rank in its span's list of every vertex after a first.
    uint2* node;
    uint32_t* node_rank;
    uint32_t node_cap, rank_cap;
};

__device__ __forceinline__ uint32_t lanes_below(uint32_t n) {  // bits of lanes 0 .. n - 1
    return n >= 32u ? FULL : (1u << n) - 1u;
}

// ---- heap (every lane calls with the same arguments) -------------------------------------------

__device__ __noinline__ void* heap_alloc(WarpHeap& h, size_t bytes) {
    const uint64_t words = ((uint64_t)bytes + 15u) / 16u * 4u;
    const uint32_t lo = h.lo, top = h.top;
    uint32_t* p = nullptr;
    uint32_t nlo = lo, ntop = top;
    if (words <= h.lo_end - lo) {
        p = h.w + lo;
        nlo = lo + (uint32_t)words;
    } else if (words <= h.cap - top) {
        p = h.w + top;
        ntop = top + (uint32_t)words;
    }
    __syncwarp();
    if ((threadIdx.x & 31) == 0) {
        h.lo = nlo;
        h.top = ntop;
    }
    __syncwarp();
    return p;
}
// A block that nothing uses any more: kept for reuse if it is the larger one.
__device__ __noinline__ void heap_free(WarpHeap& h, const void* block, size_t bytes) {
    __syncwarp();
    const uintptr_t base = reinterpret_cast<uintptr_t>(h.w), at = reinterpret_cast<uintptr_t>(block);
    const bool inside = at >= base && at < base + (uintptr_t)h.top * 4u;  // not in shared memory
    const uint32_t off = (uint32_t)((at - base) / 4u);
    const uint32_t words = (uint32_t)((bytes + 15u) / 16u * 4u);
    const bool larger = words > h.lo_end - h.lo;
    __syncwarp();
    if ((threadIdx.x & 31) == 0 && inside && larger) {
        h.lo = off;
        h.lo_end = off + words;
    }
    __syncwarp();
}
template <class T>
__device__ __forceinline__ T* heap_array(WarpHeap& h, uint32_t n) {
    return static_cast<T*>(heap_alloc(h, (size_t)n * sizeof(T)));
}
// Room for `want` elements; false when the heap has none.
template <class T>
__device__ __noinline__ bool grow_array(WarpHeap& h, T*& p, uint32_t n, uint32_t& cap, uint32_t want) {
    uint32_t nc = cap * 2u;
    if (nc < want) nc = want;
    T* q = heap_array<T>(h, nc);
    if (!q) return false;
    const T* old = p;
#pragma unroll 1
    for (uint32_t i = threadIdx.x & 31; i < n; i += 32) q[i] = old[i];
    heap_free(h, old, (size_t)cap * sizeof(T));
    p = q;
    cap = nc;
    return true;
}

// grow_array of a member of SweepSmem.
template <class T>
__device__ __noinline__ bool grow_member(WarpHeap& h, T** p, uint32_t n, uint32_t* cap, uint32_t want) {
    T* q = *p;
    uint32_t c = *cap;
    const bool ok = grow_array(h, q, n, c, want);
    __syncwarp();
    if ((threadIdx.x & 31) == 0) {
        *p = q;
        *cap = c;
    }
    __syncwarp();
    return ok;
}
__device__ __noinline__ bool grow_uids(SweepSmem& S, uint32_t n, uint32_t want) {
    return grow_member(S.heap, &S.span_first, n, &S.uid_cap, want) &&
           grow_member(S.heap, &S.span_len, n, &S.len_cap, want) &&
           grow_member(S.heap, &S.flushed, n, &S.flushed_cap, want);
}
__device__ __noinline__ bool grow_nodes(SweepSmem& S, uint32_t n, uint32_t want) {
    return grow_member(S.heap, &S.node, n, &S.node_cap, want) &&
           grow_member(S.heap, &S.node_rank, n, &S.rank_cap, want);
}

// The next n elements of a block that is handed out piece by piece.
template <class T>
__device__ __forceinline__ T* take(char*& at, uint32_t n) {
    T* p = reinterpret_cast<T*>(at);
    at += ((size_t)n * sizeof(T) + 15u) & ~(size_t)15u;
    return p;
}
// First arrays of a path of n events, from one block.
template <bool SRC>
__device__ __noinline__ bool alloc_lists(SweepSmem& S, uint32_t n) {
    const uint32_t nv = (n + 11u) & ~3u, nn = (2 * n + 11u) & ~3u, nu = (n / 4 + 11u) & ~3u;
    const uint32_t ns = (3 * n + 27u) & ~3u;
    size_t bytes = (size_t)nv * sizeof(V2) + (size_t)nn * (sizeof(uint2) + 4u) +
                   (size_t)nu * (sizeof(float4) + sizeof(uint2) + 4u);
    if (SRC) bytes += (size_t)nv * 4u + (size_t)ns * 4u;
    char* at = static_cast<char*>(heap_alloc(S.heap, bytes));
    if (!at) return false;
    if ((threadIdx.x & 31) == 0) {
        S.span_first = take<float4>(at, nu);
        S.out_v = take<V2>(at, nv);
        S.node = take<uint2>(at, nn);
        S.span_len = take<uint2>(at, nu);
        S.node_rank = take<uint32_t>(at, nn);
        S.flushed = take<uint32_t>(at, nu);
        S.out_sfirst = SRC ? take<uint32_t>(at, nv) : nullptr;
        S.out_src = SRC ? take<uint32_t>(at, ns) : nullptr;
        S.out_cap = nv;
        S.node_cap = S.rank_cap = nn;
        S.uid_cap = S.len_cap = S.flushed_cap = nu;
        S.sfirst_cap = SRC ? nv : 0u;
        S.src_cap = SRC ? ns : 0u;
    }
    __syncwarp();
    return true;
}

// ---- event queue -------------------------------------------------------------------------------

template <bool SRC>
__device__ __noinline__ bool alloc_events(WarpHeap& h, Events& ev, uint32_t cap) {
    cap = (cap + 3u) & ~3u;
    const size_t per = sizeof(float4) + sizeof(V2) + sizeof(uint32_t) + sizeof(uint2) +
                       (SRC ? sizeof(uint2) : 0);
    char* at = static_cast<char*>(heap_alloc(h, per * cap));
    if (!at) return false;
    if ((threadIdx.x & 31) == 0) {
        ev.edge = take<float4>(at, cap);
        ev.pos = take<V2>(at, cap);
        ev.wind = take<uint32_t>(at, cap);
        ev.link = take<uint2>(at, cap);
        ev.ids = SRC ? take<uint2>(at, cap) : nullptr;
        ev.cap = cap;
    }
    __syncwarp();
    return true;
}
// Room for `want` events, keeping the first n.
template <bool SRC>
__device__ __noinline__ bool grow_events(SweepSmem& S, uint32_t n, uint32_t want) {
    const Events o = S.ev;
    __syncwarp();
    uint32_t cap = o.cap * 2u;
    if (cap < want) cap = want;
    if (!alloc_events<SRC>(S.heap, S.ev, cap)) return false;
    const Events e = S.ev;
#pragma unroll 1
    for (uint32_t i = threadIdx.x & 31; i < n; i += 32) {
        e.pos[i] = o.pos[i];
        e.edge[i] = o.edge[i];
        e.wind[i] = o.wind[i];
        e.link[i] = o.link[i];
        if (SRC) e.ids[i] = o.ids[i];
    }
    heap_free(S.heap, o.edge, (size_t)o.cap * (sizeof(float4) + sizeof(V2) + sizeof(uint32_t) +
                                               sizeof(uint2) + (SRC ? sizeof(uint2) : 0)));
    return true;
}
__device__ __forceinline__ uint32_t pack_wind(int32_t winding, bool is_edge) {
    return ((uint32_t)winding & 0xFFFFu) | (is_edge ? IS_EDGE : 0u);
}
template <bool SRC>
__device__ __forceinline__ void put_event(const Events& e, uint32_t i, V2 pos, V2 to, float t0,
                                          float t1, uint32_t wind, uint32_t from_id,
                                          uint32_t to_id) {
    e.pos[i] = pos;
    e.edge[i] = make_float4(to.x, to.y, t0, t1);
    e.wind[i] = wind;
    if (SRC) e.ids[i] = make_uint2(from_id, to_id);
}

struct InsertArgs {
    V2 pos;
    EdgeData d;
    uint32_t after, from_id, to_id;
    uint32_t rank;     // events [0, rank] of the sorted ones are behind the sweep
    uint32_t sibling;  // insert_sibling (event_queue.rs:215-230) of this event, NONE: by position
};
// event_queue.rs:188-274: appends an event and links it into the list. lyon walks the list from
// `after`; every event of [rank + 1, sorted_n) is further down the list, in order, so the walk
// starts at the last of them that is not past the position. Returns the event, NONE without room.
template <bool SRC>
__device__ __noinline__ uint32_t insert_event(SweepSmem& S, const InsertArgs& A) {
    const uint32_t lane = threadIdx.x & 31;
    __syncwarp();
    const uint32_t idx = S.ev.n;
    if (idx >= S.ev.cap && !grow_events<SRC>(S, idx, idx + 1)) return NONE;
    const Events e = S.ev;
    __syncwarp();
    if (lane == 0) {
        put_event<SRC>(e, idx, A.pos, A.d.to, A.d.range_start, A.d.range_end,
                       pack_wind(A.d.winding, A.d.is_edge != 0), A.from_id, A.to_id);
        e.link[idx] = make_uint2(NONE, NONE);
        S.ev.n = idx + 1;
    }
    __syncwarp();
    if (A.sibling != NONE) {
        if (lane == 0) {
            e.link[idx].x = e.link[A.sibling].x;
            e.link[A.sibling].x = idx;
        }
        __syncwarp();
        return idx;
    }
    uint32_t start = A.after;
    const uint32_t n = S.sorted_n;
    if (n > 0 && A.rank + 1 < n) {
        // The first sorted event that is not before the position: 32 probes at a time.
        uint32_t lo = A.rank + 1, hi = n;
#pragma unroll 1
        while (lo < hi) {
            const uint32_t step = (hi - lo + 31u) / 32u;
            const uint32_t i = lo + lane * step;
            const bool before = i < hi && is_after(A.pos, e.pos[i]);
            const uint32_t m = __ballot_sync(FULL, before);
            const uint32_t c = (uint32_t)__popc(m);  // probes 0 .. c - 1 are before it
            if (c == 0) {
                hi = lo;
                break;
            }
            const uint32_t nhi = lo + c * step;
            lo = lo + (c - 1u) * step + 1u;
            if (nhi < hi) hi = nhi;
        }
        uint32_t c = lo;
        if (!(c < n && peq(e.pos[c], A.pos))) {
            c = c - 1u;  // the head of the events before it
#pragma unroll 1
            while (c > A.rank && peq(e.pos[c - 1u], e.pos[c])) --c;
        }
        if (c > A.rank && !peq(e.pos[c], e.pos[A.rank])) start = c;
    }
    uint32_t prev = start, current = start;
#pragma unroll 1
    for (;;) {
        if (current == NONE) {
            __syncwarp();
            if (lane == 0) e.link[prev].y = idx;
            break;
        }
        const V2 pos = e.pos[current];
        const uint2 l = e.link[current];
        if (peq(pos, A.pos)) {
            __syncwarp();
            if (lane == 0) {
                e.link[idx].x = l.x;
                e.link[current].x = idx;
            }
            break;
        }
        if (is_after(pos, A.pos)) {
            __syncwarp();
            if (lane == 0) {
                e.link[prev].y = idx;
                e.link[idx].y = current;
            }
            break;
        }
        prev = current;
        current = l.y;
    }
    __syncwarp();
    return idx;
}

// event_queue.rs:301-395: lyon's merge sort on linked lists, step by step (lane 0). Only for
// queues with a NaN position, whose order is what those steps make of it.
__device__ __noinline__ uint32_t merge_sort_lists(const Events& E) {
    const V2* pos = E.pos;
    uint2* link = E.link;
    auto merge = [&](uint32_t a, uint32_t b) -> uint32_t {
        if (a == NONE) return b;
        if (b == NONE) return a;
        bool first_node = true;
        uint32_t sorted_head = NONE, prev = NONE;
#pragma unroll 1
        for (;;) {
            if (a == NONE) {
                if (!first_node) link[prev].y = b;
                break;
            }
            if (b == NONE) {
                if (!first_node) link[prev].y = a;
                break;
            }
            uint32_t node;
            const int c = compare_positions(pos[a], pos[b]);
            if (c < 0) {
                node = a;
                a = link[a].y;
            } else if (c > 0) {
                node = b;
                b = link[b].y;
            } else {
                uint32_t s = a;  // find_last_sibling (event_queue.rs:386-395)
#pragma unroll 1
                while (link[s].x != NONE) s = link[s].x;
                link[s].x = b;
                b = link[b].y;
                continue;
            }
            if (first_node) {
                first_node = false;
                sorted_head = node;
            } else {
                link[prev].y = node;
            }
            prev = node;
        }
        if (sorted_head == NONE) sorted_head = a;
        return sorted_head;
    };
    struct Frame {
        uint32_t s, e, stage, a;
    };
    Frame stk[40];
    int sp = 0;
    uint32_t ret = 0;
    stk[sp++] = Frame{0, E.n, 0, 0};
#pragma unroll 1
    while (sp > 0) {
        Frame& f = stk[sp - 1];
        const uint32_t split = (f.s + f.e) / 2;
        if (f.stage == 0) {
            if (split == f.s) {
                ret = f.s;
                --sp;
                continue;
            }
            f.stage = 1;
            stk[sp++] = Frame{f.s, split, 0, 0};
        } else if (f.stage == 1) {
            f.a = ret;
            f.stage = 2;
            stk[sp++] = Frame{split, f.e, 0, 0};
        } else {
            ret = merge(f.a, ret);
            --sp;
        }
    }
    return ret;
}

// A float's order as an unsigned word, -0 as +0.
__device__ __forceinline__ uint32_t ordered(float f) {
    const uint32_t u = f2u(f == 0.0f ? 0.0f : f);
    return u ^ ((u >> 31) ? 0xFFFFFFFFu : 0x80000000u);
}

// Orders the queue (event_queue.rs:301-395): S.ev becomes a copy in order of position, events of
// one position next to each other in the order in which they were made, as lyon's merges chain
// them; links set. The old arrays and the scratch become the heap's room to reuse. Returns the
// first event; *oom on a full heap.
template <bool SRC>
__device__ __noinline__ uint32_t sort_events(SweepSmem& S, uint32_t lo, bool* oom) {
    const uint32_t lane = threadIdx.x & 31;
    const Events o = S.ev;
    const uint32_t n = o.n;
    *oom = false;
    if (n == 0) return NONE;
    bool nan = false;
#pragma unroll 1
    for (uint32_t i = lane; i < n; i += 32) {
        const V2 p = o.pos[i];
        nan = nan || p.x != p.x || p.y != p.y;
    }
    if (__any_sync(FULL, nan)) {
#pragma unroll 1
        for (uint32_t i = lane; i < n; i += 32) o.link[i] = make_uint2(NONE, NONE);
        __syncwarp();
        uint32_t first = 0;
        if (lane == 0) first = merge_sort_lists(S.ev);
        __syncwarp();
        return __shfl_sync(FULL, first, 0);
    }
    if (n <= 32) {  // a lane per event, in place
        const bool live = lane < n;
        V2 p = V2{0.0f, 0.0f};
        float4 edge = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        uint32_t wind = 0;
        uint2 ids = make_uint2(0u, 0u);
        unsigned long long k = ~0ull;
        if (live) {
            p = o.pos[lane];
            edge = o.edge[lane];
            wind = o.wind[lane];
            if (SRC) ids = o.ids[lane];
            k = ((unsigned long long)ordered(p.y) << 32) | ordered(p.x);
        }
        uint32_t r = 0;
        bool tie = false;  // with an event made before
#pragma unroll 1
        for (uint32_t j = 0; j < n; ++j) {
            const unsigned long long q = __shfl_sync(FULL, k, (int)j);
            r += q < k || (q == k && j < lane) ? 1u : 0u;
            tie = tie || (q == k && j < lane);
        }
        __syncwarp();
        if (live) {
            o.pos[r] = p;
            o.edge[r] = edge;
            o.wind[r] = wind;
            if (SRC) o.ids[r] = ids;
        }
        // Bit r: the event at place r is the first of its position.
        uint32_t heads = live && !tie ? 1u << r : 0u;
        for (uint32_t d = 16; d > 0; d /= 2) heads |= __shfl_xor_sync(FULL, heads, d);
        if (live) {
            const uint32_t above = lane == 31 ? 0u : heads & (FULL << (lane + 1));
            const bool next_is_head = lane + 1 >= n || ((heads >> (lane + 1)) & 1u) != 0;
            o.link[lane] = make_uint2(next_is_head ? NONE : lane + 1,
                                      above ? (uint32_t)__ffs((int)above) - 1u : NONE);
        }
        if (lane == 0) S.sorted_n = n;
        __syncwarp();
        return 0;
    }
    unsigned long long* key = heap_array<unsigned long long>(S.heap, n);
    unsigned long long* key2 = heap_array<unsigned long long>(S.heap, n);
    uint32_t* id = heap_array<uint32_t>(S.heap, n);
    uint32_t* id2 = heap_array<uint32_t>(S.heap, n);
    if (!key || !key2 || !id || !id2) {
        *oom = true;
        return NONE;
    }
    // Runs of 32, ranked by counting.
#pragma unroll 1
    for (uint32_t base = 0; base < n; base += 32) {
        const uint32_t i = base + lane;
        unsigned long long k = ~0ull;
        if (i < n) {
            const V2 p = o.pos[i];
            k = ((unsigned long long)ordered(p.y) << 32) | ordered(p.x);
        }
        const uint32_t m = n - base < 32u ? n - base : 32u;
        uint32_t r = 0;
#pragma unroll 1
        for (uint32_t j = 0; j < m; ++j) {
            const unsigned long long q = __shfl_sync(FULL, k, (int)j);
            r += q < k || (q == k && j < lane) ? 1u : 0u;
        }
        if (i < n) {
            key[base + r] = k;
            id[base + r] = i;
        }
    }
    __syncwarp();
    // Merges: an element's place is its own index in its run and the number of elements of the
    // other run before it (of the left run also those equal to it).
#pragma unroll 1
    for (uint32_t run = 32; run < n; run *= 2) {
        // Four elements per lane, so that four searches' loads are on their way at a time.
#pragma unroll 1
        for (uint32_t base = lane; base < n; base += 128) {
            unsigned long long k[4];
            uint32_t other[4], len[4], c[4];  // the other run, its length, how many are before
            bool left[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t i = base + 32u * u;
                const uint32_t pair = i & ~(2 * run - 1u);
                left[u] = i < pair + run;
                other[u] = left[u] ? pair + run : pair;
                len[u] = i >= n || other[u] >= n ? 0u : n - other[u] < run ? n - other[u] : run;
                c[u] = 0;
                k[u] = i < n ? key[i] : 0ull;
            }
#pragma unroll 1
            for (uint32_t width = run; width > 0; width /= 2) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint32_t probe = c[u] + width;
                    if (probe <= len[u]) {
                        const unsigned long long q = key[other[u] + probe - 1u];
                        if (q < k[u] || (!left[u] && q == k[u])) c[u] = probe;
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t i = base + 32u * u;
                if (i < n) {
                    const uint32_t at = (left[u] ? i : i - run) + c[u];
                    key2[at] = k[u];
                    id2[at] = id[i];
                }
            }
        }
        __syncwarp();
        unsigned long long* tk = key;
        key = key2;
        key2 = tk;
        uint32_t* ti = id;
        id = id2;
        id2 = ti;
        if (run > 0x40000000u) break;
    }
    // The copy, with room for the events that intersections add.
    const uint32_t cap = n + n / 8 + 16;
    if (!alloc_events<SRC>(S.heap, S.ev, cap)) {
        *oom = true;
        return NONE;
    }
    const Events e = S.ev;
    uint32_t next_head = NONE;  // the first head after the chunk
#pragma unroll 1
    for (uint32_t base = (n - 1) / 32 * 32;; base -= 32) {
        const uint32_t i = base + lane;
        bool head = false, next_is_head = true;
        if (i < n) {
            const uint32_t j = id[i];
            const V2 p = o.pos[j];
            e.pos[i] = p;
            e.edge[i] = o.edge[j];
            e.wind[i] = o.wind[j];
            if (SRC) e.ids[i] = o.ids[j];
            head = i == 0 || key[i - 1] != key[i];
            next_is_head = i + 1 >= n || key[i + 1] != key[i];
        }
        const uint32_t heads = __ballot_sync(FULL, head);
        const uint32_t above = lane == 31 ? 0u : heads & (FULL << (lane + 1));
        if (i < n) {
            const uint32_t nh = above ? base + (uint32_t)__ffs((int)above) - 1u : next_head;
            e.link[i] = make_uint2(next_is_head ? NONE : i + 1, nh);
        }
        if (heads) next_head = base + (uint32_t)__ffs((int)heads) - 1u;
        if (base == 0) break;
    }
    __syncwarp();
    if (lane == 0) {
        S.sorted_n = n;
        // The copy was allocated last: all between `lo` and it is free.
        S.heap.lo = lo;
        S.heap.lo_end = (uint32_t)(reinterpret_cast<uint32_t*>(e.edge) - S.heap.w);
    }
    __syncwarp();
    return 0;
}

// ---- monotone tessellators (monotone.rs), a span per lane ----------------------------------------

// The vertex list of a span: nodes[0] is the vertex it began at; x, y, and the id with the side in
// bit 31 (lists are ordered as the sweep made them). Writes the triangles to `out` (null: only
// counts them) and returns their number. ev: two lists of k + 1 ids, stk: k + 1 words.
__device__ __noinline__ uint32_t tessellate_span(const float4* nodes, uint32_t k, bool ended,
                                                 uint32_t* ev_l, uint32_t* ev_r, uint32_t* stk,
                                                 uint32_t* out) {
    struct Side {
        V2 ref;
        float cx;
        V2 prev, last;
        uint32_t last_node, n;
        uint32_t* ev;
    };
    const float4 b4 = nodes[0];
    const V2 bp = V2{b4.x, b4.y};
    const uint32_t bid = f2u(b4.z) & 0x7FFFFFFFu;
    Side sd[2];
    for (int i = 0; i < 2; ++i) {
        sd[i].ref = bp;
        sd[i].cx = bp.x;
        sd[i].prev = V2{0.0f, 0.0f};  // side_push: the position of the empty `last`
        sd[i].last = bp;
        sd[i].last_node = 0;
        sd[i].n = 1;
        sd[i].ev = i == LEFT ? ev_l : ev_r;
        sd[i].ev[0] = bid;
    }
    uint32_t tris = 0;
    uint32_t sn = 1;  // the basic tessellator's stack (monotone.rs:9-139)
    stk[0] = 0;
    uint32_t prev_node = 0;
    int prev_side = LEFT;
    auto tri = [&](uint32_t a, uint32_t b, uint32_t c) {
        if (out) {
            out[3 * (size_t)tris] = a;
            out[3 * (size_t)tris + 1] = b;
            out[3 * (size_t)tris + 2] = c;
        }
        ++tris;
    };
    float4 next = k > 1 ? nodes[1] : b4;
#pragma unroll 1
    for (uint32_t j = 1; j < k; ++j) {
        const float4 c4 = next;
        if (j + 1 < k) next = nodes[j + 1];
        const V2 pos = V2{c4.x, c4.y};
        const uint32_t id = f2u(c4.z) & 0x7FFFFFFFu;
        const int side = (int)(f2u(c4.z) >> 31);
        const bool end = ended && j + 1 == k;
        // Steps: of a vertex (monotone.rs:263-330) the flush of the opposite side and of its own,
        // each followed by the flushed side's last vertex; of the end (monotone.rs:332-359) both
        // flushes, then their vertices in order of position, then the end itself.
        int f0 = -1, f1 = -1, steps = 0;
        if (end) {
            f0 = LEFT;
            f1 = RIGHT;
            steps = 5;
        } else {
            Side& s = sd[side];
            Side& opp = sd[1 - side];
            if (side == LEFT) {
                s.ref.x = fmaxf(s.ref.x, pos.x);
                s.cx = fmaxf(s.cx, s.ref.x);
            } else {
                s.ref.x = fminf(s.ref.x, pos.x);
                s.cx = fminf(s.cx, s.ref.x);
            }
            const float dx = sd[RIGHT].cx - sd[LEFT].cx;
            const float dy = pos.y - s.ref.y;
            const bool sides_are_close = dx < dy * 0.1f;
            bool outward_turn = false;
            if (!sides_are_close && s.n >= 2) {
                const float sign = side == LEFT ? 1.0f : -1.0f;
                outward_turn = cross(s.prev - s.last, pos - s.last) * sign < 0.0f;
            }
            if (outward_turn || sides_are_close) {
                if (is_after(s.last, opp.last)) f0 = 1 - side;
                f1 = side;
                steps = 2;
            }
        }
        uint32_t va = NONE, vb = NONE;
#pragma unroll 1
        for (int step = 0; step < steps; ++step) {
            const int f = step == 0 ? f0 : step == 1 ? f1 : -1;
            uint32_t v = NONE;
            if (f >= 0 && sd[f].n >= 2) {
                // monotone.rs:362-404
                Side& s = sd[f];
                const uint32_t* ev = s.ev;
                const uint32_t len = s.n;
#pragma unroll 1
                for (uint32_t st = 1; st * 2 < len; st *= 2) {
                    uint32_t last_index = 0;
                    const uint32_t imax = (len - 1) / (2 * st);
#pragma unroll 1
                    for (uint32_t i = 0; i < imax; ++i) {
                        const uint32_t a = ev[last_index], b = ev[last_index + st];
                        last_index += 2 * st;
                        const uint32_t c = ev[last_index];
                        tri(f == RIGHT ? b : a, f == RIGHT ? a : b, c);
                    }
                    if (last_index + st < len) {
                        const uint32_t b = ev[last_index], c = ev[last_index + st];
                        tri(ev[0], f == RIGHT ? c : b, f == RIGHT ? b : c);
                    }
                }
                s.ev[0] = ev[len - 1];
                s.n = 1;
                s.prev = s.last;
                s.ref = s.last;
                v = s.last_node;
                if (!end) {
                    // The other side's reference becomes exact again.
                    Side& q = sd[1 - f];
                    q.cx = q.ref.x;
                }
            }
            if (end) {
                if (step == 0) {
                    va = v;
                    continue;
                }
                if (step == 1) {
                    vb = v;
                    if (va != NONE && vb != NONE && is_after(sd[LEFT].last, sd[RIGHT].last)) {
                        const uint32_t t = va;
                        va = vb;
                        vb = t;
                    }
                    continue;
                }
                v = step == 2 ? va : step == 3 ? vb : j;
            }
            if (v == NONE) continue;
            // BasicMonotoneTessellator (monotone.rs:53-139)
            const float4 v4 = nodes[v];
            const V2 vp = V2{v4.x, v4.y};
            const uint32_t vid = f2u(v4.z) & 0x7FFFFFFFu;
            const int vside = end && step == 4 ? 1 - prev_side : (int)(f2u(v4.z) >> 31);
            if (vside != prev_side) {
                float4 a4 = nodes[stk[0]];
#pragma unroll 1
                for (uint32_t i = 0; i + 1 < sn; ++i) {
                    const float4 n4 = nodes[stk[i + 1]];
                    const V2 a = V2{a4.x, a4.y}, b = V2{n4.x, n4.y};
                    const uint32_t ia = f2u(a4.z) & 0x7FFFFFFFu, ib = f2u(n4.z) & 0x7FFFFFFFu;
                    const bool winding = cross(a - b, vp - b) >= 0.0f;
                    tri(winding ? ia : ib, winding ? ib : ia, vid);
                    a4 = n4;
                }
                stk[0] = prev_node;
                sn = 1;
            } else if (sn > 0) {
                uint32_t last_popped = stk[--sn];
                bool have_last = true;
                float4 l4 = nodes[last_popped];
#pragma unroll 1
                while (sn > 0) {
                    const uint32_t t = stk[sn - 1];
                    const float4 t4 = nodes[t];
                    const float4 a4 = vside == RIGHT ? t4 : l4, q4 = vside == RIGHT ? l4 : t4;
                    const V2 a = V2{a4.x, a4.y}, b = V2{q4.x, q4.y};
                    if (!(cross(vp - b, a - b) >= 0.0f)) break;
                    tri(f2u(q4.z) & 0x7FFFFFFFu, f2u(a4.z) & 0x7FFFFFFFu, vid);
                    have_last = sn > 0;
                    if (have_last) {
                        last_popped = stk[--sn];
                        l4 = nodes[last_popped];
                    }
                }
                if (have_last) stk[sn++] = last_popped;
            }
            stk[sn++] = v;
            prev_node = v;
            prev_side = vside;
        }
        if (!end) {  // monotone.rs:202-209
            Side& s = sd[side];
            s.ev[s.n++] = id;
            s.prev = s.last;
            s.last = pos;
            s.last_node = j;
        }
    }
    return tris;
}

// ---- error recovery: the order of the active edges (fill.rs:1848-1955), lane 0 -------------------

__device__ __noinline__ bool sort_active_edges(float4* A, uint4* B, uint32_t n, float* K,
                                               uint32_t* O, float4* SA, uint4* SB, V2 current,
                                               int fill_rule) {
    const float y = current.y;
    bool has_merge_vertex = false;
    float prev_x = u2f(0x7fc00000u);
#pragma unroll 1
    for (uint32_t i = 0; i < n; ++i) {
        const V2 from = ae_from(A[i]), to = ae_to(A[i]);
        float key;
        if (ae_is_merge(B[i])) {
            has_merge_vertex = true;
            key = prev_x;
        } else {
            const bool eq_to = to.y == y, eq_from = from.y == y;
            float x;
            if (eq_to && eq_from) {
                const float current_x = current.x;
                x = (max_x(from, to) >= current_x && min_x(from, to) <= current_x)
                        ? current.x
                        : min_x(from, to);
            } else if (eq_from) {
                x = from.x;
            } else if (eq_to) {
                x = to.x;
            } else {
                x = solve_x_for_y(from, to, y);
            }
            key = fmax_lyon(x, min_x(from, to));
            prev_x = x;
        }
        K[i] = key;
        O[i] = i;
    }
    if (n > 1) {
#pragma unroll 1
        for (uint32_t i = 0; i < n; ++i)
            if (K[i] != K[i]) return false;  // lyon unwraps a NaN comparison here
    }
    auto key_less = [&](float ka, uint32_t ia, float kb, uint32_t ib) {
        if (ka < kb) return true;
        if (ka > kb) return false;
        const bool ma = ae_is_merge(B[ia]), mb = ae_is_merge(B[ib]);
        if (!ma && !mb)
            return slope(ae_to(A[ib]) - ae_from(A[ib])) < slope(ae_to(A[ia]) - ae_from(A[ia]));
        return !ma && mb;
    };
#pragma unroll 1
    for (uint32_t i = 1; i < n; ++i) {  // stable insertion sort (Vec::sort_by is stable)
        uint32_t j = i;
#pragma unroll 1
        while (j > 0 && key_less(K[j], O[j], K[j - 1], O[j - 1])) {
            const float tk = K[j];
            K[j] = K[j - 1];
            K[j - 1] = tk;
            const uint32_t to = O[j];
            O[j] = O[j - 1];
            O[j - 1] = to;
            --j;
        }
    }
#pragma unroll 1
    for (uint32_t i = 0; i < n; ++i) {
        SA[i] = A[O[i]];
        SB[i] = B[O[i]];
    }
#pragma unroll 1
    for (uint32_t i = 0; i < n; ++i) {
        A[i] = SA[i];
        B[i] = SB[i];
    }
    if (!has_merge_vertex) return true;
    int16_t winding_number = 0;
#pragma unroll 1
    for (uint32_t i = 0; i < n; ++i) {
        bool needs_swap;
        if (ae_is_merge(B[i])) {
            needs_swap = !fill_rule_is_in(fill_rule, winding_number);
        } else {
            winding_number = w16(winding_number + ae_winding(B[i]));
            needs_swap = false;
        }
        if (needs_swap) {
            int16_t w = winding_number;
            uint32_t idx = i;
#pragma unroll 1
            while (idx > 0) {
                w = w16(w - ae_winding(B[idx - 1]));
                const float4 ta = A[idx];
                A[idx] = A[idx - 1];
                A[idx - 1] = ta;
                const uint4 tb = B[idx];
                B[idx] = B[idx - 1];
                B[idx - 1] = tb;
                if (fill_rule_is_in(fill_rule, w)) break;
                idx -= 1;
            }
        }
    }
    return true;
}

// The number of steps of a curve (of a quadratic with c2 unused).
__device__ __noinline__ float curve_steps(bool cubic, V2 from, V2 c1, V2 c2, V2 to, float tol) {
    return cubic ? cubic_wang(from, c1, c2, to, tol) : quad_wang(from, c1, to, tol);
}

// ---- a path --------------------------------------------------------------------------------------

// The warp's state of the path it sweeps: uniform over the lanes, in registers but for `S`. SRC:
// the fill also records every vertex's sources (an instantiation of its own).
template <bool SRC>
struct WarpFiller {
    SweepSmem& S;
    const uint32_t lane;
    int err;  // 0, a LYON_ERR_* code, or FILL_ERR_HEAP
    int fill_rule, orientation;
    float tolerance;
    bool assume_no_intersection;
    uint32_t out_n, src_n;
    // Sweep line
    float4* act_a;
    uint4* act_b;
    uint32_t act_n, act_cap;
    WarpPending* below;
    uint32_t below_n, below_cap;
    // Live spans in order: uid, length of the vertex list.
    uint2* spans;
    uint32_t spans_n, spans_cap;
    uint32_t nuid, node_n, flushed_n;
    V2 pos;            // the current event
    uint32_t vertex;   // its output vertex
    uint32_t event, rank;
    bool relink;       // an event was added (or one's range changed) since the next was loaded
    // Active edge scan (fill.rs:115-151). Vertex events: at most two; spans to end: successive.
    int32_t ve_span0, ve_span1;
    int ve_side0;
    uint32_t ve_n;
    int32_t end_first;
    uint32_t end_n;
    bool sc_merge_event, sc_split_event, any_split;
    uint32_t above_start, above_end;
    WindingState before_point;

    __device__ __forceinline__ WarpFiller(SweepSmem& s) : S(s), lane(threadIdx.x & 31) {}

    __device__ __forceinline__ void fail(int code) {
        if (err == 0) err = code;
    }
    template <class T>
    __device__ __forceinline__ bool room(T*& p, uint32_t n, uint32_t& cap, uint32_t want) {
        if (want <= cap) return true;
        T* q = p;  // (only the copies' addresses are taken)
        uint32_t c = cap;
        const bool ok = grow_array(S.heap, q, n, c, want);
        if (!ok) fail(FILL_ERR_HEAP);
        p = q;
        cap = c;
        return ok;
    }

    // ---- spans ----
    __device__ __forceinline__ void begin_span(int32_t idx, V2 position, uint32_t id) {
        if (idx < 0 || (uint32_t)idx > spans_n) {
            fail(LYON_ERR_INTERNAL);
            return;
        }
        if (!room(spans, spans_n, spans_cap, spans_n + 1)) return;
        if (nuid >= S.flushed_cap && !grow_uids(S, nuid, nuid + 1)) {
            fail(FILL_ERR_HEAP);
            return;
        }
        insert_span((uint32_t)idx);
        if (lane == 0) {
            spans[idx] = make_uint2(nuid, 1u);
            S.span_first[nuid] = make_float4(position.x, position.y, u2f(id), 0.0f);
            S.span_len[nuid] = make_uint2(0u, 0u);
        }
        __syncwarp();
        ++nuid;
        ++spans_n;
    }
    __device__ __forceinline__ void insert_span(uint32_t idx) {  // moves [idx, n) up by one
        uint32_t hi = spans_n;
#pragma unroll 1
        while (hi > idx) {
            const uint32_t c = hi - idx < 32u ? hi - idx : 32u;
            const uint32_t i = hi - c + lane;
            uint2 v = make_uint2(0u, 0u);
            if (lane < c) v = spans[i];
            __syncwarp();
            if (lane < c) spans[i + 1] = v;
            __syncwarp();
            hi -= c;
        }
    }
    // Appends the current vertex to a live span's list.
    __device__ __forceinline__ void add_to_span(int32_t idx, int side) {
        if (idx < 0 || (uint32_t)idx >= spans_n) {
            fail(LYON_ERR_INTERNAL);
            return;
        }
        if (node_n >= S.rank_cap && !grow_nodes(S, node_n, node_n + 1)) {
            fail(FILL_ERR_HEAP);
            return;
        }
        const uint2 s = spans[idx];
        __syncwarp();
        if (lane == 0) {
            S.node[node_n] = make_uint2(s.x, vertex | ((uint32_t)side << 31));
            S.node_rank[node_n] = s.y;
            spans[idx].y = s.y + 1u;
        }
        __syncwarp();
        ++node_n;
    }
    __device__ __forceinline__ void flush_span(uint2 s, bool ended) {
        if (lane == 0) {
            S.span_len[s.x].x = s.y;
            S.flushed[flushed_n] = s.x | (ended ? 0u : 0x80000000u);
        }
        __syncwarp();
        ++flushed_n;
    }

    // ---- active edge scan (fill.rs:1045-1378) ----
    __device__ __forceinline__ void before_edges_done(const WindingState& winding, uint32_t idx,
                                                      bool previous_was_merge, bool connecting) {
        above_start = idx;
        before_point = winding;
        bool merge_split = false;
        if (previous_was_merge) {
            before_point.span_index -= 1;
            above_start -= 1;
            if (!connecting) {
                ve_span0 = winding.span_index - 1;
                ve_side0 = RIGHT;
                ve_span1 = winding.span_index;
                ve_n = 2;
                merge_split = true;
            }
        }
        sc_split_event = !connecting && winding.is_in && !merge_split;
    }
    __device__ __forceinline__ void connecting_edges_done(const WindingState& winding,
                                                          bool in_before_vertex) {
        const bool in_after_vertex = winding.is_in;
        if (in_before_vertex && in_after_vertex && below_n == 0 && !any_split)
            sc_merge_event = true;
        if (in_before_vertex) {
            ve_span0 = before_point.span_index;
            ve_side0 = RIGHT;
            ve_n = 1;
        }
        if (in_after_vertex) {
            if (ve_n) {
                ve_span1 = winding.span_index;
            } else {
                ve_span0 = winding.span_index;
                ve_side0 = LEFT;
            }
            ve_n += 1;
        }
    }
    // False: lyon's ActiveEdgeScan error (recovered from by ordering the edges anew). Every lane
    // answers lyon's questions about its edge, the walk along the edges is done on the answers'
    // ballots.
    __device__ __forceinline__ bool scan_active_edges() {
        ve_n = 0;
        end_n = 0;
        end_first = 0;
        sc_merge_event = sc_split_event = any_split = false;
        const float cx = pos.x, thr = tolerance;
        bool prev_merge = false, in_before = false, first_connecting = false;
        int phase = 0;  // 0: edges before the point; 1: edges connecting to it; 2: the rest
        uint32_t idx = 0;
        WindingState winding;  // (its number: in front of the chunk)
        winding.reset();
#pragma unroll 1
        for (uint32_t base = 0; base < act_n; base += 32) {
            const uint32_t live_n = act_n - base < 32u ? act_n - base : 32u;
            const bool live = lane < live_n;
            float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            uint32_t bw = 0;
            if (live) {
                a = act_a[base + lane];
                bw = act_b[base + lane].x;
            }
            const V2 from = ae_from(a), to = ae_to(a);
            const bool merge = (bw & AE_MERGE) != 0;
            const bool edge = live && !merge;
            const int32_t w = (int32_t)(int16_t)(bw & 0xFFFFu);
            const float lo = min_x(from, to), hi = max_x(from, to);
            const bool at_to = peq(pos, to), horizontal = from.y == to.y;
            const float ex = solve_x_for_y(from, to, pos.y);
            const bool left = hi < cx, right = lo > cx, near = fabsf(ex - cx) <= thr;
            // The edge is before the point, or connects to it (fill.rs:1085-1125).
            const bool before = !at_to && (left || (!right && !horizontal && !near && !(ex > cx)));
            const bool conn = at_to || (!left && !right && (horizontal || near));
            // Among the connecting edges (fill.rs:1328-1378).
            const bool passed = hi + thr < cx || to.y < pos.y;
            const float x = !horizontal ? ex : hi >= cx && lo <= cx ? cx : to.x;
            const bool close = fabsf(x - cx) <= thr;
            const bool one = at_to || (!passed && !right && close);
            const bool bad = !at_to && (passed || (!right && !close && x < cx));
            // Among the remaining ones (fill.rs:1295-1324).
            const bool wrong = left || at_to || (lo < cx && ex < cx);
            const uint32_t m_merge = __ballot_sync(FULL, merge);
            const uint32_t m_edge = __ballot_sync(FULL, edge);
            const uint32_t m_after = __ballot_sync(FULL, edge && !before);
            const uint32_t m_conn = __ballot_sync(FULL, conn);
            const uint32_t m_other = __ballot_sync(FULL, edge && !one);
            const uint32_t m_split = __ballot_sync(FULL, edge && one && !at_to);
            const uint32_t m_bad = __ballot_sync(FULL, bad);
            const uint32_t m_wrong = __ballot_sync(FULL, edge && wrong);
            // The winding number behind every lane.
            const uint32_t m_up = __ballot_sync(FULL, edge && w == 1);
            const uint32_t m_down = __ballot_sync(FULL, edge && w == -1);
            const uint32_t m_wide = __ballot_sync(FULL, edge && (w > 1 || w < -1));
            const uint32_t le = FULL >> (31u - lane);
            int32_t num = __popc(m_up & le) - __popc(m_down & le);
            if (m_wide) {
                num = edge ? w : 0;
#pragma unroll 1
                for (uint32_t d = 1; d < 32; d *= 2) {
                    const int32_t o = __shfl_up_sync(FULL, num, d);
                    if (lane >= d) num += o;
                }
            }
            const int16_t n16 = w16(winding.number + num);
            const uint32_t m_in = __ballot_sync(FULL, edge && fill_rule_is_in(fill_rule, n16));
            uint32_t at = 0;  // first lane of the phase
            if (phase == 0) {
                const uint32_t f = m_after ? (uint32_t)__ffs((int)m_after) - 1u : live_n;
                const uint32_t m_f = lanes_below(f), m_e = m_edge & m_f;
                winding.span_index += __popc(m_in & m_f) + __popc(m_merge & m_f);
                if (m_e) winding.is_in = ((m_in >> (31 - __clz((int)m_e))) & 1u) != 0;
                if (f > 0) prev_merge = ((m_merge >> (f - 1u)) & 1u) != 0;
                idx = base + f;
                if (m_after) {
                    const int16_t number = winding.number;
                    if (m_wide) {
                        const int n = __shfl_sync(FULL, (int)n16, m_e ? 31 - __clz((int)m_e) : 0);
                        if (m_e) winding.number = (int16_t)n;
                    } else {
                        winding.number = w16(number + __popc(m_up & m_f) - __popc(m_down & m_f));
                    }
                    const bool connecting = ((m_conn >> f) & 1u) != 0;
                    before_edges_done(winding, idx, prev_merge, connecting);
                    winding.number = number;
                    in_before = winding.is_in;
                    first_connecting = !prev_merge;
                    phase = connecting ? 1 : 2;
                    at = f;
                }
            }
            if (phase == 1) {
                const uint32_t rest = FULL << at;
                const uint32_t stop = m_other & rest;
                const uint32_t t = stop ? (uint32_t)__ffs((int)stop) - 1u : live_n;
                if (m_split & rest & lanes_below(t)) any_split = true;
#pragma unroll 1
                for (uint32_t l = at; l < t; ++l) {
                    const bool m = ((m_merge >> l) & 1u) != 0;
                    if (m && !winding.is_in) return false;  // MergeVertexOutside
                    if (m || (!first_connecting && winding.is_in)) {
                        if (end_n == 0) end_first = winding.span_index;
                        ++end_n;
                    }
                    if (!m) winding.is_in = ((m_in >> l) & 1u) != 0;
                    if (m || winding.is_in) winding.span_index += 1;
                    if (!m && winding.is_in && winding.span_index >= (int32_t)spans_n) return false;
                    first_connecting = false;
                }
                idx = base + t;
                if (stop) {
                    if ((m_bad >> t) & 1u) return false;
                    connecting_edges_done(winding, in_before);
                    phase = 2;
                    at = t;
                }
            }
            if (phase == 2 && (m_wrong & (FULL << at))) return false;
            winding.number = (int16_t)__shfl_sync(FULL, (int)n16, 31);
        }
        if (phase == 0) before_edges_done(winding, idx, prev_merge, false);
        if (phase == 1) connecting_edges_done(winding, in_before);
        above_end = idx;
        return true;
    }

    // ---- edges above / below the current point (fill.rs:1381-1524) ----
    __device__ __forceinline__ void add_below(V2 to, uint32_t src, int32_t winding,
                                              float range_end) {
        if (!room(below, below_n, below_cap, below_n + 1)) return;
        if (lane == 0) {
            WarpPending e;
            e.to = to;
            e.sort_key = 0.0f;  // sort_edges_below, when there is another edge
            e.range_end = range_end;
            e.src_edge = src;
            e.winding = winding;
            e.pad[0] = e.pad[1] = 0;
            below[below_n] = e;
        }
        __syncwarp();
        ++below_n;
    }
    __device__ __forceinline__ void process_edges_above() {
        // The vertex joins the lists of the vertex events' spans, then ends those to end: a lane
        // each. A span that is met twice takes it twice.
        const bool twice = ve_n > 1 && ve_span0 == ve_span1;
#pragma unroll 1
        for (uint32_t base = 0; base < ve_n + end_n; base += 32) {
            const uint32_t i = base + lane;
            const bool live = i < ve_n + end_n, end = i >= ve_n;
            const int32_t idx = end ? end_first + (int32_t)(i - ve_n) : i == 0 ? ve_span0 : ve_span1;
            const bool ends = idx >= end_first && idx - end_first < (int32_t)end_n;
            if (__any_sync(FULL, live && (idx < 0 || (uint32_t)idx >= spans_n))) {
                fail(LYON_ERR_INTERNAL);
                return;
            }
            if (node_n + 32 > S.rank_cap && !grow_nodes(S, node_n, node_n + 32)) {
                fail(FILL_ERR_HEAP);
                return;
            }
            if (live) {
                const uint2 s = spans[idx];
                const uint32_t again = (ve_n > 0 && i > 0 && idx == ve_span0 ? 1u : 0u) +
                                       (ve_n > 1 && i > 1 && idx == ve_span1 ? 1u : 0u);
                const int side = i == 0 && !end ? ve_side0 : LEFT;
                S.node[node_n + lane] = make_uint2(s.x, vertex | ((uint32_t)side << 31));
                S.node_rank[node_n + lane] = s.y + again;
                if (end) {
                    S.span_len[s.x].x = s.y + again + 1u;
                    S.flushed[flushed_n + i - ve_n] = s.x;
                } else if (!ends && !twice) {
                    spans[idx].y = s.y + 1u;
                }
            }
            node_n += ve_n + end_n - base < 32u ? ve_n + end_n - base : 32u;
            __syncwarp();
        }
        // (Both lanes have read the span: one of them cannot write it before.)
        if (twice && (ve_span0 < end_first || ve_span0 - end_first >= (int32_t)end_n)) {
            if (lane == 0) spans[ve_span0].y += 2u;
            __syncwarp();
        }
        flushed_n += end_n;
        if (end_n > 0) {
#pragma unroll 1
            for (uint32_t i = (uint32_t)end_first + end_n; i < spans_n; i += 32) {
                uint2 v = make_uint2(0u, 0u);
                const bool live = i + lane < spans_n;
                if (live) v = spans[i + lane];
                __syncwarp();
                if (live) spans[i + lane - end_n] = v;
                __syncwarp();
            }
            spans_n -= end_n;
        }
        if (any_split) {
#pragma unroll 1
            for (uint32_t i = above_start; i < above_end; ++i) {
                const float4 a = act_a[i];
                const uint4 b = act_b[i];
                if (ae_is_merge(b) || peq(pos, ae_to(a))) continue;
                add_below(ae_to(a), b.z, ae_winding(b), u2f(b.w));
                if (err) return;
                if (lane == 0) act_a[i] = make_float4(a.x, a.y, pos.x, pos.y);
                __syncwarp();
            }
        }
        if (sc_merge_event) {
            const float4 a = act_a[above_start];
            const uint4 b = act_b[above_start];
            __syncwarp();
            if (lane == 0) {
                act_a[above_start] = make_float4(a.z, a.w, a.z, a.w);
                act_b[above_start] = make_uint4(AE_MERGE, vertex, b.z, b.w);
            }
            __syncwarp();
            above_start += 1;
        }
    }
    __device__ __forceinline__ uint32_t insert_sorted(V2 p, const EdgeData& d, uint2 ids,
                                                      uint32_t sibling = NONE) {
        InsertArgs A;
        A.pos = p;
        A.d = d;
        A.after = event;
        A.from_id = ids.x;
        A.to_id = ids.y;
        A.rank = rank;
        A.sibling = sibling;
        relink = true;
        const uint32_t e = insert_event<SRC>(S, A);
        if (e == NONE) fail(FILL_ERR_HEAP);
        return e;
    }
    __device__ __forceinline__ uint2 ids_of(uint32_t e) {
        return SRC ? S.ev.ids[e] : make_uint2(LYON_NO_ENDPOINT, LYON_NO_ENDPOINT);
    }
    // fill.rs:2010-2013 (sort_unstable_by on the sort key; insertion order for short slices)
    __device__ __forceinline__ void sort_edges_below() {
#pragma unroll 1
        for (uint32_t i = lane; i < below_n; i += 32) below[i].sort_key = slope(below[i].to - pos);
        __syncwarp();
        if (lane == 0) {
#pragma unroll 1
            for (uint32_t i = 1; i < below_n; ++i) {
                uint32_t j = i;
#pragma unroll 1
                while (j > 0 && below[j].sort_key < below[j - 1].sort_key) {
                    const WarpPending t = below[j];
                    below[j] = below[j - 1];
                    below[j - 1] = t;
                    --j;
                }
            }
        }
        __syncwarp();
    }
    __device__ __forceinline__ void merge_coincident_edges(uint32_t a_idx, uint32_t b_idx) {  // fill.rs:2050-2106
        const V2 a_to = below[a_idx].to, b_to = below[b_idx].to;
        const int c = compare_positions(a_to, b_to);
        const uint32_t lower_idx = c < 0 ? b_idx : a_idx, upper_idx = c < 0 ? a_idx : b_idx;
        const WarpPending edge = below[lower_idx];
        const V2 split_point = below[upper_idx].to;
        const int32_t w = w16(below[upper_idx].winding + edge.winding);
        __syncwarp();
        if (lane == 0) {
            below[upper_idx].winding = w;
#pragma unroll 1
            for (uint32_t k = lower_idx; k + 1 < below_n; ++k) below[k] = below[k + 1];
        }
        __syncwarp();
        --below_n;
        if (c == 0) return;
        const float range_start = S.ev.edge[edge.src_edge].z;
        const float dy = edge.to.y - pos.y;
        const float t = dy == 0.0f ? 0.0f : (split_point.y - pos.y) / dy;
        const float t_remapped = remap_t_in_range(t, range_start, edge.range_end);
        insert_sorted(split_point, EdgeData{edge.to, t_remapped, edge.range_end, edge.winding, 1u},
                      ids_of(edge.src_edge));
    }
    __device__ __forceinline__ void handle_coincident_edges_below() {  // fill.rs:2016-2048
#pragma unroll 1
        for (int idx = (int)below_n - 2; idx >= 0; --idx) {
            const uint32_t a_idx = (uint32_t)idx, b_idx = a_idx + 1;
            const float a_slope = below[a_idx].sort_key;
            const float b_slope = below[b_idx].sort_key;
            const float THRESHOLD = 0.00005f;
            bool angle_is_close;
            if (fabsf(a_slope) <= 1.0f) {
                angle_is_close = fabsf(a_slope - b_slope) < THRESHOLD;
            } else {
                angle_is_close = fabsf(1.0f / a_slope - 1.0f / b_slope) < THRESHOLD;
            }
            if (angle_is_close) {
                merge_coincident_edges(a_idx, b_idx);
                if (err) return;
            }
        }
    }
    __device__ __forceinline__ void split_event(uint32_t left_idx, int32_t left_span_idx) {  // fill.rs:1563-1608
        const uint32_t right_idx = left_idx + 1;
        if (right_idx >= act_n) {
            fail(LYON_ERR_INTERNAL);
            return;
        }
        const V2 lf = ae_from(act_a[left_idx]), rf = ae_from(act_a[right_idx]);
        const bool left = is_after(lf, rf);
        const uint32_t upper_id = left ? act_b[left_idx].y : act_b[right_idx].y;
        begin_span(left ? left_span_idx : left_span_idx + 1, left ? lf : rf, upper_id);
#pragma unroll 1
        for (int i = 0; i < 2 && err == 0; ++i)
            add_to_span(left_span_idx + i, i == 0 ? RIGHT : LEFT);
    }
    __device__ __forceinline__ void process_edges_below() {  // fill.rs:1455-1524
        WindingState winding = before_point;
        if (below_n > 1) {
            sort_edges_below();
            handle_coincident_edges_below();
            if (err) return;
        }
        if (sc_split_event) {
            if (above_start == 0) {
                fail(LYON_ERR_INTERNAL);
                return;
            }
            split_event(above_start - 1, winding.span_index);
            if (err) return;
        }
#pragma unroll 1
        for (uint32_t i = 0; i + 1 < below_n; ++i) {
            winding.update(fill_rule, w16(below[i].winding));
            if (winding.is_in) {
                begin_span(winding.span_index, pos, vertex);
                if (err) return;
            }
        }
    }

    // ---- intersections (fill.rs:1611-1846) ----
    __device__ __forceinline__ void process_intersection(double ta, double tb, uint32_t ai,
                                                         uint32_t bi) {
        const WarpPending eb = below[bi];
        const float4 a4 = act_a[ai];
        const uint4 a_b = act_b[ai];
        const V2 a_from = ae_from(a4), a_to = ae_to(a4);
        const float a_end = u2f(a_b.w);
        const int32_t a_wind = ae_winding(a_b);
        const double bfx = pos.x, bfy = pos.y, btx = eb.to.x, bty = eb.to.y;
        const double one_t = 1.0 - tb;
        V2 ip = V2{(float)(one_t * bfx + tb * btx), (float)(one_t * bfy + tb * bty)};
        const float a_start = S.ev.edge[a_b.z].z;
        if (peq(pos, ip)) {
            __syncwarp();
            if (lane == 0) {
                act_a[ai] = make_float4(ip.x, ip.y, a4.z, a4.w);
                S.ev.edge[a_b.z].z = remap_t_in_range((float)ta, a_start, a_end);
            }
            __syncwarp();
            relink = true;
            return;
        }
        if (!is_after(ip, pos)) ip.y = nextafterf(pos.y, INFINITY);
        if (!is_after(ip, pos)) {
            fail(LYON_ERR_INTERNAL);  // lyon asserts here
            return;
        }
        if (is_near(ip, eb.to)) {
            ip = eb.to;
        } else if (is_near(ip, a_to)) {
            ip = a_to;
        }
        const float b_start = S.ev.edge[eb.src_edge].z;
        const uint2 a_ids = ids_of(a_b.z), b_ids = ids_of(eb.src_edge);
        uint32_t inserted_evt = NONE;
        bool flipped_active = false;
        if (!peq(a_to, ip) && !peq(a_from, ip)) {
            const float remapped_ta = remap_t_in_range((float)ta, a_start, a_end);
            const bool below_ip = is_after(a_to, ip);
            flipped_active = !below_ip;
            const uint32_t e = insert_sorted(
                below_ip ? ip : a_to,
                below_ip ? EdgeData{a_to, remapped_ta, a_end, a_wind, 1u}
                         : EdgeData{ip, a_end, remapped_ta, (int32_t)w16(-a_wind), 1u},
                a_ids);
            if (err) return;
            if (below_ip) inserted_evt = e;
            if (lane == 0) {
                act_a[ai] = make_float4(a_from.x, a_from.y, ip.x, ip.y);
                act_b[ai] = make_uint4(a_b.x, a_b.y, a_b.z, f2u(remapped_ta));
            }
            __syncwarp();
        }
        if (!peq(eb.to, ip) && !peq(pos, ip)) {
            const float remapped_tb = remap_t_in_range((float)tb, b_start, eb.range_end);
            const bool below_ip = is_after(eb.to, ip);
            insert_sorted(below_ip ? ip : eb.to,
                          below_ip ? EdgeData{eb.to, remapped_tb, eb.range_end, eb.winding, 1u}
                                   : EdgeData{ip, eb.range_end, remapped_tb,
                                              (int32_t)w16(-eb.winding), 1u},
                          b_ids, below_ip ? inserted_evt : NONE);
            if (err) return;
            if (!below_ip && flipped_active) {  // event_queue.rs:232-250
                insert_sorted(ip,
                              EdgeData{V2{u2f(0x7fc00000u), u2f(0x7fc00000u)}, 0.0f, 0.0f, 0, 0u},
                              make_uint2(b_ids.y, b_ids.y));
                if (err) return;
            }
            if (lane == 0) {
                below[bi].to = ip;
                below[bi].range_end = remapped_tb;
            }
            __syncwarp();
        }
    }
    __device__ __forceinline__ void handle_intersections() {
        const uint32_t skip_start = above_start, skip_end = above_end;
#pragma unroll 1
        for (uint32_t bi = 0; bi < below_n; ++bi) {
            const V2 bt = below[bi].to;
            const float below_min_x = fminf(pos.x, bt.x);
            const float below_max_x = fmax_lyon(pos.x, bt.x);
            // The first of the intersections nearest to the point (the least tb): each lane keeps
            // the first of its edges.
            double tb_min = 1.0, fta = 0.0;
            uint32_t fidx = NONE;
#pragma unroll 1
            for (uint32_t base = 0; base < act_n; base += 32) {
                const uint32_t i = base + lane;
                bool may = i < act_n && !(i >= skip_start && i < skip_end);
                float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (may) {
                    a = act_a[i];
                    may = !ae_is_merge(act_b[i]);
                }
                const V2 from = ae_from(a), to = ae_to(a);
                may = may && !(below_min_x > max_x(from, to)) && !(below_max_x < min_x(from, to)) &&
                      !share_end_point(from, to, pos, bt);
                if (!__any_sync(FULL, may)) continue;
                may = may && may_intersect(from, to, pos, bt);
                double ta, tb;
                if (may && intersection_t(from, to, pos, bt, &ta, &tb)) {
                    if (tb < tb_min && tb > 0.0 && ta > 0.0 && ta <= 1.0) {
                        tb_min = tb;
                        fta = ta;
                        fidx = i;
                    }
                }
            }
            uint32_t m = __ballot_sync(FULL, fidx != NONE);
            if (!m) continue;
            double best_tb = 0.0, best_ta = 0.0;
            uint32_t best = NONE;
#pragma unroll 1
            while (m) {
                const int l = __ffs((int)m) - 1;
                m &= m - 1u;
                const double tb = __shfl_sync(FULL, tb_min, l), ta = __shfl_sync(FULL, fta, l);
                const uint32_t i = __shfl_sync(FULL, fidx, l);
                if (best == NONE || tb < best_tb || (tb == best_tb && i < best)) {
                    best = i;
                    best_tb = tb;
                    best_ta = ta;
                }
            }
            process_intersection(best_ta, best_tb, best, bi);
            if (err) return;
        }
    }
    __device__ __forceinline__ void update_active_edges() {  // fill.rs:1527-1561
        if (!assume_no_intersection) {
            handle_intersections();
            if (err) return;
        }
        const uint32_t s = above_start, e = above_end, gone = e - s, nb = below_n;
        const uint32_t new_n = act_n - gone + nb;
        if (new_n > act_cap &&
            (!grow_active(new_n))) {
            return;
        }
        if (nb > gone) {  // the edges after the point move up
            const uint32_t by = nb - gone;
            uint32_t hi = act_n;
#pragma unroll 1
            while (hi > e) {
                const uint32_t c = hi - e < 32u ? hi - e : 32u;
                const uint32_t i = hi - c + lane;
                float4 a;
                uint4 b;
                if (lane < c) {
                    a = act_a[i];
                    b = act_b[i];
                }
                __syncwarp();
                if (lane < c) {
                    act_a[i + by] = a;
                    act_b[i + by] = b;
                }
                __syncwarp();
                hi -= c;
            }
        } else if (nb < gone) {
            const uint32_t by = gone - nb;
#pragma unroll 1
            for (uint32_t lo = e; lo < act_n; lo += 32) {
                const uint32_t i = lo + lane;
                float4 a;
                uint4 b;
                if (i < act_n) {
                    a = act_a[i];
                    b = act_b[i];
                }
                __syncwarp();
                if (i < act_n) {
                    act_a[i - by] = a;
                    act_b[i - by] = b;
                }
                __syncwarp();
            }
        }
#pragma unroll 1
        for (uint32_t k = lane; k < nb; k += 32) {
            const WarpPending p = below[k];
            act_a[s + k] = make_float4(pos.x, pos.y, p.to.x, p.to.y);
            act_b[s + k] = make_uint4((uint32_t)p.winding & 0xFFFFu, vertex, p.src_edge,
                                      f2u(p.range_end));
        }
        __syncwarp();
        act_n = new_n;
        below_n = 0;
    }
    __device__ __forceinline__ bool grow_active(uint32_t want) {
        uint32_t cap = act_cap;
        if (!room(act_a, act_n, cap, want)) return false;
        return room(act_b, act_n, act_cap, want);
    }

    // ---- error recovery (fill.rs:1848-2007) ----
    __device__ __forceinline__ void recover_from_error() {
        {
            const uint32_t lo = S.heap.lo, top = S.heap.top;
            const uint32_t n = act_n;
            float* keys = heap_array<float>(S.heap, n);
            uint32_t* order = heap_array<uint32_t>(S.heap, n);
            float4* sa = heap_array<float4>(S.heap, n);
            uint4* sb = heap_array<uint4>(S.heap, n);
            if (!keys || !order || !sa || !sb) {
                fail(FILL_ERR_HEAP);
                return;
            }
            int sorted = 1;
            if (lane == 0) {
                sorted = sort_active_edges(act_a, act_b, n, keys, order, sa, sb, pos, fill_rule);
                S.heap.lo = lo;
                S.heap.top = top;
            }
            __syncwarp();
            if (!__shfl_sync(FULL, sorted, 0)) {
                fail(LYON_ERR_INTERNAL);
                return;
            }
        }
        const uint32_t len = act_n;
        if (len > 1 && lane == 0 && ae_is_merge(act_b[len - 1])) {
            const float4 ta = act_a[len - 1];
            act_a[len - 1] = act_a[len - 2];
            act_a[len - 2] = ta;
            const uint4 tb = act_b[len - 1];
            act_b[len - 1] = act_b[len - 2];
            act_b[len - 2] = tb;
        }
        __syncwarp();
        WindingState winding;
        winding.reset();
#pragma unroll 1
        for (uint32_t i = 0; i < act_n; ++i) {
            const uint4 b = act_b[i];
            if (ae_is_merge(b)) {
                winding.span_index += 1;
            } else {
                winding.update(fill_rule, w16(ae_winding(b)));
            }
            if (winding.span_index >= (int32_t)spans_n) {
                begin_span(winding.span_index, ae_from(act_a[i]), b.y);
                if (err) return;
            }
        }
#pragma unroll 1
        while ((int64_t)spans_n > (int64_t)winding.span_index + 1) {
            flush_span(spans[spans_n - 1], false);
            spans_n -= 1;
        }
    }

    // VertexSourceIterator (fill.rs:2294-2337): every sibling event at the vertex gives its
    // edge's endpoint (t = 0 or 1) or the point at t on it; a source equal to the previous one is
    // skipped.
    __device__ __forceinline__ void record_sources(uint32_t ev) {
        if (out_n >= S.sfirst_cap &&
            !grow_member(S.heap, &S.out_sfirst, out_n, &S.sfirst_cap, out_n + 1)) {
            fail(FILL_ERR_HEAP);
            return;
        }
        if (lane == 0) S.out_sfirst[out_n] = src_n;
        uint32_t pf = 0, pt = 0;
        float ptt = 0.0f;
        bool have_prev = false;
#pragma unroll 1
        for (uint32_t id = ev; id != NONE; id = S.ev.link[id].x) {
            const float t = S.ev.edge[id].z;
            const uint2 e = S.ev.ids[id];
            uint32_t f = e.x, to = LYON_NO_ENDPOINT;
            float tt = 0.0f;
            if (t == 1.0f) {
                f = e.y;
            } else if (t != 0.0f) {
                to = e.y;
                tt = t;
            }
            if (have_prev && f == pf && to == pt && (to == LYON_NO_ENDPOINT || tt == ptt)) continue;
            if (3 * src_n + 3 > S.src_cap &&
                !grow_member(S.heap, &S.out_src, 3 * src_n, &S.src_cap, 3 * src_n + 3)) {
                fail(FILL_ERR_HEAP);
                return;
            }
            if (lane == 0) {
                uint32_t* d = S.out_src + 3 * (size_t)src_n;
                d[0] = f;
                d[1] = to;
                d[2] = f2u(tt);
            }
            ++src_n;
            pf = f;
            pt = to;
            ptt = tt;
            have_prev = true;
        }
        __syncwarp();
    }

    // ---- main loop (fill.rs:749-965) ----
    __device__ __forceinline__ void tessellator_loop(uint32_t first) {
        event = first;
        if (event == NONE) return;
        V2 n_pos = S.ev.pos[event];
        uint2 n_link = S.ev.link[event];
        float4 n_edge = S.ev.edge[event];
        uint32_t n_wind = S.ev.wind[event];
        rank = 0;
#pragma unroll 1
        while (event != NONE) {
            pos = n_pos;
            const float4 edge = n_edge;
            const uint32_t wind = n_wind;
            const uint2 link = n_link;
            relink = false;
            if (event < S.sorted_n) rank = event;
            if (link.y != NONE) {  // the next event, on its way while this one is worked on
                n_pos = S.ev.pos[link.y];
                n_edge = S.ev.edge[link.y];
                n_wind = S.ev.wind[link.y];
                n_link = S.ev.link[link.y];
            }
            if (pos.x != pos.x || pos.y != pos.y) {
                fail(LYON_ERR_POSITION_IS_NAN);
                return;
            }
            if (SRC) record_sources(event);
            if (out_n >= S.out_cap &&
                !grow_member(S.heap, &S.out_v, out_n, &S.out_cap, out_n + 1)) {
                fail(FILL_ERR_HEAP);
                return;
            }
            if (lane == 0)
                S.out_v[out_n] =
                    orientation == LYON_ORIENTATION_VERTICAL ? pos : V2{pos.y, -pos.x};
            vertex = out_n++;
            uint32_t sib = event, w = wind, next = link.x;
            float4 d = edge;
#pragma unroll 1
            for (;;) {
                if (w & IS_EDGE)
                    add_below(V2{d.x, d.y}, sib, (int32_t)(int16_t)(w & 0xFFFFu), d.w);
                sib = next;
                if (sib == NONE) break;
                w = S.ev.wind[sib];
                d = S.ev.edge[sib];
                next = S.ev.link[sib].x;
            }
            if (err) return;
            bool recovered = false;
#pragma unroll 1
            while (!scan_active_edges()) {
                if (recovered) {
                    fail(LYON_ERR_INTERNAL);
                    return;
                }
                recover_from_error();
                if (err) return;
                recovered = true;
            }
            process_edges_above();
            if (err) return;
            process_edges_below();
            if (err) return;
            update_active_edges();
            if (err) return;
            if (relink) {
                const uint32_t next = S.ev.link[event].y;
                event = next;
                if (next != NONE) {
                    n_pos = S.ev.pos[next];
                    n_edge = S.ev.edge[next];
                    n_wind = S.ev.wind[next];
                    n_link = S.ev.link[next];
                }
            } else {
                event = link.y;
            }
        }
    }

    // ---- event queue construction (event_queue.rs:441-905) ----
    struct Builder {
        V2 current, prev, second;
        uint32_t nth;
        uint32_t prev_id;  // prev_endpoint_id
        float tolerance;
        uint32_t n;  // events
    };
    __device__ __forceinline__ bool event_room(uint32_t n, uint32_t want) {
        if (want <= S.ev.cap) return true;
        if (grow_events<SRC>(S, n, want)) return true;
        fail(FILL_ERR_HEAP);
        return false;
    }
    __device__ __forceinline__ void eq_vertex_event(Builder& b, V2 at, uint32_t id) {
        if (!event_room(b.n, b.n + 1)) return;
        if (lane == 0) {
            const V2 nan = V2{u2f(0x7fc00000u), u2f(0x7fc00000u)};
            put_event<SRC>(S.ev, b.n, at, nan, 0.0f, 0.0f, pack_wind(0, false), id, id);
        }
        b.n += 1;
    }
    __device__ __forceinline__ void eq_line_segment(Builder& b, V2 to, uint32_t to_id) {
        const V2 from = b.current;
        if (peq(from, to)) return;
        const bool up = is_after(from, to);
        if (up && b.nth > 0 && is_after(from, b.prev)) eq_vertex_event(b, from, b.prev_id);
        if (b.nth == 0) b.second = to;
        if (!event_room(b.n, b.n + 1)) return;
        if (lane == 0)
            put_event<SRC>(S.ev, b.n, up ? to : from, up ? from : to, up ? 1.0f : 0.0f,
                           up ? 0.0f : 1.0f, pack_wind(up ? -1 : 1, true), b.prev_id, to_id);
        b.n += 1;
        b.nth += 1;
        b.prev = b.current;
        b.prev_id = to_id;
        b.current = to;
    }
    // Shared body of quadratic_bezier_segment / cubic_bezier_segment (event_queue.rs:758-900):
    // the (possibly swapped) segment flattened with lyon's for_each_flattened_with_t, a point per
    // lane. A swapped curve's t values are those of the swapped segment while its ids stay the
    // original ones.
    __device__ __forceinline__ void eq_curve(Builder& b, V2 original_from, V2 original_to,
                                             uint32_t to_id, bool needs_swap, const Poly& poly,
                                             V2 seg_from, V2 seg_to, float n) {
        const int32_t winding = needs_swap ? -1 : 1;
        V2 prev_pt = seg_from, first_pt = V2{0.0f, 0.0f};
        bool have_first = false;
        const bool is_first_edge = b.nth == 0;
        // flatten_with_t: count = to_u32(n) - 1 interior steps, t += 1/n, then the end point.
        const float step = 1.0f / n;
        const uint32_t count = to_u32_or1(n) - 1;
        float t_before = 0.0f;   // of the point before the chunk
        V2 p_before = seg_from;
#pragma unroll 1
        for (uint32_t base = 0; base <= count && base <= 0xFFFFFFDFu; base += 32) {
            const uint32_t m = count - base < 32u ? count - base + 1u : 32u;  // points here
            float t1 = t_before;
#pragma unroll 1
            for (uint32_t j = 0; j < m; ++j)
                if (j <= lane) t1 = t1 + step;
            V2 to = poly_sample(poly, t1);
            if (base + lane == count) {
                t1 = 1.0f;
                to = seg_to;
            }
            float t0 = __shfl_up_sync(FULL, t1, 1);
            V2 from = V2{__shfl_up_sync(FULL, to.x, 1), __shfl_up_sync(FULL, to.y, 1)};
            if (lane == 0) {
                t0 = t_before;
                from = p_before;
            }
            const bool valid = lane < m && !peq(from, to);
            const uint32_t m_valid = __ballot_sync(FULL, valid);
            const uint32_t m_before = m_valid & lanes_below(lane);
            // The point before the edge before this one.
            const int pl = m_before ? 31 - __clz((int)m_before) : 0;
            V2 pp = V2{__shfl_sync(FULL, from.x, pl), __shfl_sync(FULL, from.y, pl)};
            if (!m_before) pp = prev_pt;
            const bool up = is_after(from, to);
            const bool corner =
                valid && (have_first || m_before) && up && is_after(from, pp);
            const uint32_t m_corner = __ballot_sync(FULL, corner);
            if (!event_room(b.n, b.n + (uint32_t)(__popc(m_valid) + __popc(m_corner)))) return;
            if (valid) {
                uint32_t at =
                    b.n + (uint32_t)(__popc(m_before) + __popc(m_corner & lanes_below(lane)));
                if (corner) {
                    const V2 nan = V2{u2f(0x7fc00000u), u2f(0x7fc00000u)};
                    put_event<SRC>(S.ev, at, from, nan, t0, t0, pack_wind(0, false), b.prev_id,
                                   to_id);
                    ++at;
                }
                put_event<SRC>(S.ev, at, up ? to : from, up ? from : to, up ? t1 : t0,
                               up ? t0 : t1, pack_wind(up ? -winding : winding, true), b.prev_id,
                               to_id);
            }
            b.n += (uint32_t)(__popc(m_valid) + __popc(m_corner));
            if (m_valid) {
                const int fl = __ffs((int)m_valid) - 1, ll = 31 - __clz((int)m_valid);
                const V2 fp = V2{__shfl_sync(FULL, to.x, fl), __shfl_sync(FULL, to.y, fl)};
                if (!have_first) first_pt = fp;
                have_first = true;
                prev_pt = V2{__shfl_sync(FULL, from.x, ll), __shfl_sync(FULL, from.y, ll)};
                b.nth += (uint32_t)__popc(m_valid);
            }
            t_before = __shfl_sync(FULL, t1, 31);
            p_before = V2{__shfl_sync(FULL, to.x, 31), __shfl_sync(FULL, to.y, 31)};
        }
        if (have_first) {
            const V2 second_pt = needs_swap ? prev_pt : first_pt;
            const V2 previous = needs_swap ? first_pt : prev_pt;
            if (is_first_edge) {
                b.second = second_pt;
            } else if (is_after(original_from, b.prev) && is_after(original_from, second_pt)) {
                eq_vertex_event(b, original_from, b.prev_id);
            }
            b.prev = previous;
            b.current = original_to;
            b.prev_id = to_id;
        }
    }
    __device__ __forceinline__ static uint32_t verb_points(uint32_t v) {
        return v == LYON_VERB_QUADRATIC_TO ? 2u : v == LYON_VERB_CUBIC_TO ? 3u
               : v == LYON_VERB_END ? 0u : 1u;
    }
    // Lane's verb of the window at `base`, and the index of its first point (both passes below).
    __device__ __forceinline__ uint32_t window_verb(const uint8_t* verbs, uint32_t nverbs,
                                                    uint32_t base, uint32_t& pi, uint32_t& first,
                                                    uint32_t& np) {
        const bool live = base + lane < nverbs;
        const uint32_t v = live ? verbs[base + lane] : 0u;
        np = live ? verb_points(v) : 0u;
        uint32_t incl = np;
        for (uint32_t d = 1; d < 32; d *= 2) {
            const uint32_t o = __shfl_up_sync(FULL, incl, d);
            if (lane >= d) incl += o;
        }
        first = pi + incl - np;
        pi += __shfl_sync(FULL, incl, 31);
        return v;
    }
    // Number of edges the event queue builder will produce at most (lines, flattened curve
    // segments, closing edges); an estimate for reservations only. False for a malformed path
    // (unknown verbs, missing points).
    __device__ __forceinline__ bool count_segments(const uint8_t* verbs, uint32_t nverbs,
                                                   const float* pts, uint32_t npts,
                                                   float tol, uint32_t* total) {
        uint32_t segs = 0, pi = 0;
#pragma unroll 1
        for (uint32_t base = 0; base < nverbs; base += 32) {
            uint32_t first, np;
            const uint32_t v = window_verb(verbs, nverbs, base, pi, first, np);
            const bool bad = v > LYON_VERB_END || (np > 0 && first + np > npts) || pi < first;
            if (__any_sync(FULL, bad)) return false;
            uint32_t s = base + lane < nverbs ? 1u : 0u;
            if (np > 1) {
                const V2 from = first > 0 ? V2{pts[2 * first - 2], pts[2 * first - 1]}
                                          : V2{0.0f, 0.0f};
                const V2 c1 = V2{pts[2 * first], pts[2 * first + 1]};
                const V2 c2 = V2{pts[2 * first + 2], pts[2 * first + 3]};
                const V2 to = np == 3 ? V2{pts[2 * first + 4], pts[2 * first + 5]} : c2;
                s = to_u32_or1(curve_steps(np == 3, from, c1, c2, to, tol));
                if (s > (1u << 20)) s = 1u << 20;
            }
            for (uint32_t d = 16; d > 0; d /= 2) s += __shfl_xor_sync(FULL, s, d);
            segs += s;
            if (segs > (1u << 20)) segs = 1u << 20;
        }
        *total = segs;
        return true;
    }
    // Builds the event queue of a path (event_queue.rs:483-551 set_path).
    __device__ __forceinline__ void build_events(const uint8_t* verbs, uint32_t nverbs,
                                                 const float* pts, const lyon_fill_options& o) {
        Builder b;
        b.current = b.prev = b.second = V2{u2f(0x7fc00000u), u2f(0x7fc00000u)};
        b.nth = 0;
        b.prev_id = LYON_NO_ENDPOINT;
        b.tolerance = o.tolerance;
        b.n = 0;
        const bool horizontal = o.sweep_orientation == LYON_ORIENTATION_HORIZONTAL;
        V2 first_pt = V2{0.0f, 0.0f};
        uint32_t first_id = LYON_NO_ENDPOINT;
        uint32_t pi = 0;
#pragma unroll 1
        for (uint32_t base = 0; base < nverbs; base += 32) {
            uint32_t first, np;
            const uint32_t v = window_verb(verbs, nverbs, base, pi, first, np);
            V2 q[3];
            for (uint32_t j = 0; j < 3; ++j) {
                q[j] = V2{0.0f, 0.0f};
                if (j < np) {
                    const V2 p = V2{pts[2 * (first + j)], pts[2 * (first + j) + 1]};
                    q[j] = horizontal ? V2{-p.y, p.x} : p;  // event_queue.rs:13-16
                }
            }
            const uint32_t m = nverbs - base < 32u ? nverbs - base : 32u;
#pragma unroll 1
            for (uint32_t l = 0; l < m; ++l) {
                const uint32_t k = __shfl_sync(FULL, v, (int)l);
                const uint32_t id0 = __shfl_sync(FULL, first, (int)l);
                const V2 p0 = V2{__shfl_sync(FULL, q[0].x, (int)l), __shfl_sync(FULL, q[0].y, (int)l)};
                if (k == LYON_VERB_QUADRATIC_TO || k == LYON_VERB_CUBIC_TO) {
                    const bool cubic = k == LYON_VERB_CUBIC_TO;
                    const V2 p1 = V2{__shfl_sync(FULL, q[1].x, (int)l),
                                     __shfl_sync(FULL, q[1].y, (int)l)};
                    const V2 p2 = V2{__shfl_sync(FULL, q[2].x, (int)l),
                                     __shfl_sync(FULL, q[2].y, (int)l)};
                    const V2 from = b.current, to = cubic ? p2 : p1;
                    const bool needs_swap = is_after(from, to);
                    const V2 sf = needs_swap ? to : from, st = needs_swap ? from : to;
                    const V2 c1 = cubic && needs_swap ? p1 : p0, c2 = needs_swap ? p0 : p1;
                    const float n = curve_steps(cubic, sf, c1, c2, st, b.tolerance);
                    const Poly poly = cubic ? cubic_poly(sf, c1, c2, st) : quad_poly(sf, c1, st);
                    eq_curve(b, from, to, id0 + (cubic ? 2u : 1u), needs_swap, poly, sf, st, n);
                } else if (k != LYON_VERB_BEGIN) {
                    const bool line = k == LYON_VERB_LINE_TO;
                    if (line || b.nth > 0) eq_line_segment(b, line ? p0 : first_pt, line ? id0 : first_id);
                    if (!line && b.nth > 0) {  // Close, End: event_queue.rs:637-659
                        if (is_after(first_pt, b.prev) && is_after(first_pt, b.second))
                            eq_vertex_event(b, first_pt, first_id);
                        b.prev_id = first_id;
                        b.nth = 0;
                    }
                } else {
                    first_pt = p0;
                    first_id = id0;
                    b.nth = 0;
                    b.current = p0;
                    b.prev_id = first_id;
                }
                if (err) return;
            }
        }
        __syncwarp();
        if (lane == 0) S.ev.n = b.n;
        __syncwarp();
    }

    // fill.rs:578-596 + 749-821: the sweep. Leaves the vertices, the spans' vertex lists and the
    // order of their flushes.
    __device__ __forceinline__ void sweep(uint32_t* heap, uint32_t heap_words,
                                          const uint8_t* verbs, uint32_t nverbs, const float* pts,
                                          uint32_t npts, const lyon_fill_options& o) {
        err = 0;
        __syncwarp();
        if (lane == 0) {
            S.heap.w = heap;
            S.heap.cap = heap_words;
            S.heap.top = S.heap.lo = S.heap.lo_end = 0;
            S.ev.n = S.ev.cap = 0;
            S.sorted_n = 0;
        }
        __syncwarp();
        out_n = src_n = act_n = below_n = spans_n = nuid = node_n = flushed_n = 0;
        act_a = S.act_a;
        act_b = S.act_b;
        act_cap = SMEM_ACTIVE;
        below = S.below;
        below_cap = SMEM_BELOW;
        spans = S.spans;
        spans_cap = SMEM_SPANS;
        // Room for every flattened edge and a vertex event per four edges, so the event arrays
        // rarely grow (a growth copies them).
        uint32_t segs = 0;
        if (!count_segments(verbs, nverbs, pts, npts, o.tolerance, &segs)) {
            fail(LYON_ERR_INVALID_ARGUMENT);
            return;
        }
        if (!alloc_events<SRC>(S.heap, S.ev, segs + segs / 4 + 8)) {
            fail(FILL_ERR_HEAP);
            return;
        }
        build_events(verbs, nverbs, pts, o);
        if (err) return;
        bool oom;
        const uint32_t first = sort_events<SRC>(S, 0, &oom);
        if (oom) {
            fail(FILL_ERR_HEAP);
            return;
        }
        const uint32_t n = S.ev.n;
        if (!alloc_lists<SRC>(S, n)) {
            fail(FILL_ERR_HEAP);
            return;
        }
        if (o.tolerance != o.tolerance || o.tolerance <= 0.0f) {
            fail(LYON_ERR_TOLERANCE_IS_NAN);
            return;
        }
        fill_rule = o.fill_rule;
        orientation = o.sweep_orientation;
        assume_no_intersection = !o.handle_intersections;
        tolerance = o.tolerance * 0.5f;
        tessellator_loop(first);
        if (err) return;
        if (assume_no_intersection && (act_n != 0 || spans_n != 0)) {
            fail(LYON_ERR_INTERNAL);
            return;
        }
#pragma unroll 1
        for (uint32_t i = 0; i < spans_n; ++i) {
            flush_span(spans[i], false);
        }
        spans_n = 0;
    }

    // The triangles of the swept path (path-relative ids): prepare_triangles lays the spans'
    // vertex lists out and returns the number of triangles, write_triangles writes them.
    float4* sorted_nodes;
    uint32_t* scratch;
    uint32_t scratch_n;
    __device__ __forceinline__ void triangulate(uint32_t f, uint32_t* out, uint32_t* count) {
        const uint32_t entry = S.flushed[f];
        const uint32_t uid = entry & 0x7FFFFFFFu;
        const uint2 len = S.span_len[uid];
        const uint32_t at = len.y + uid;
        *count = tessellate_span(sorted_nodes + len.y, len.x, !(entry >> 31), scratch + at,
                                 scratch + scratch_n + at, scratch + 2 * (size_t)scratch_n + at,
                                 out);
    }
    __device__ __forceinline__ uint32_t span_triangles(uint32_t f) {
        const uint32_t entry = S.flushed[f];
        if (!(entry >> 31)) return S.span_len[entry].x - 2u;
        uint32_t c;
        triangulate(f, nullptr, &c);
        return c;
    }
    __device__ __forceinline__ uint32_t prepare_triangles() {
        // Places of the lists, by uid.
        uint32_t total = 0;
#pragma unroll 1
        for (uint32_t base = 0; base < nuid; base += 32) {
            const uint32_t u = base + lane;
            const uint32_t k = u < nuid ? S.span_len[u].x : 0u;
            uint32_t incl = k;
            for (uint32_t d = 1; d < 32; d *= 2) {
                const uint32_t o = __shfl_up_sync(FULL, incl, d);
                if (lane >= d) incl += o;
            }
            if (u < nuid) S.span_len[u].y = total + incl - k;
            total += __shfl_sync(FULL, incl, 31);
        }
        __syncwarp();
        scratch_n = total + nuid;
        sorted_nodes = heap_array<float4>(S.heap, total);
        scratch = heap_array<uint32_t>(S.heap, 3 * scratch_n);
        if (!sorted_nodes || !scratch) {
            fail(FILL_ERR_HEAP);
            return 0;
        }
#pragma unroll 1
        for (uint32_t u = lane; u < nuid; u += 32)
            if (S.span_len[u].x) sorted_nodes[S.span_len[u].y] = S.span_first[u];
#pragma unroll 1
        for (uint32_t i = lane; i < node_n; i += 32) {
            const uint2 nd = S.node[i];
            const V2 v = S.out_v[nd.y & 0x7FFFFFFFu];
            const V2 p = orientation == LYON_ORIENTATION_VERTICAL ? v : V2{-v.y, v.x};
            sorted_nodes[S.span_len[nd.x].y + S.node_rank[i]] = make_float4(p.x, p.y, u2f(nd.y), 0.0f);
        }
        __syncwarp();
        uint32_t tris = 0;
#pragma unroll 1
        for (uint32_t base = 0; base < flushed_n; base += 32) {
            uint32_t c = base + lane < flushed_n ? span_triangles(base + lane) : 0u;
            __syncwarp();
            for (uint32_t d = 16; d > 0; d /= 2) c += __shfl_xor_sync(FULL, c, d);
            tris += c;
        }
        return tris;
    }
    __device__ __forceinline__ void write_triangles(uint32_t* out) {
        uint32_t total = 0;
#pragma unroll 1
        for (uint32_t base = 0; base < flushed_n; base += 32) {
            const bool live = base + lane < flushed_n;
            const uint32_t c = live ? span_triangles(base + lane) : 0u;
            __syncwarp();
            uint32_t incl = c;
            for (uint32_t d = 1; d < 32; d *= 2) {
                const uint32_t o = __shfl_up_sync(FULL, incl, d);
                if (lane >= d) incl += o;
            }
            uint32_t done;
            if (live && c > 0) triangulate(base + lane, out + 3 * (size_t)(total + incl - c), &done);
            __syncwarp();
            total += __shfl_sync(FULL, incl, 31);
        }
    }
};

}  // namespace fillk
}  // namespace lg
