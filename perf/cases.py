"""Cases that stand for what programs do with this library, from one path of a user interface to
the scenes of a map or a text renderer.

Every pass goes through the entry points a program calls: the one-path tessellators, the batched
calls on device memory, and the host-buffer call. Inputs are the seeded workloads of
lyon_gb300/workloads.py (curve strokes, map polylines, glyph outlines), which have the shapes and
size distributions that strokes and fills meet. A program keeps one context and reuses it for
scene after scene, so the cases share one.
"""

from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from lyon_gb300 import _native, workloads
from lyon_gb300 import tessellation as T
from lyon_gb300.options import (FILL_OPTIONS_DTYPE, STROKE_OPTIONS_DTYPE, FillOptions, FillRule,
                                LineCap, LineJoin, StrokeOptions)

CAPS = {"butt": LineCap.Butt, "square": LineCap.Square, "round": LineCap.Round}
JOINS = {"miter": LineJoin.Miter, "miter_clip": LineJoin.MiterClip, "round": LineJoin.Round,
         "bevel": LineJoin.Bevel}
RULES = {"even_odd": FillRule.EvenOdd, "non_zero": FillRule.NonZero}


def listed():
    return [
        # One shape of a user interface, stroked as lyon's tessellate_path does it: host arrays in
        # and out, one call per shape, where latency is all that counts.
        {"name": "stroke one path", "op": "path", "kind": "stroke", "segments": 16,
         "tolerance": 0.1, "join": "miter", "cap": "butt", "bits": 16},
        # One glyph filled the same way.
        {"name": "fill one glyph", "op": "path", "kind": "fill", "tolerance": 0.1,
         "rule": "non_zero", "bits": 16},
        # A scene of icons and diagrams: a thousand curve paths with 16-bit indices, each path in
        # buffers of its own.
        {"name": "stroke scene", "op": "batch", "kind": "stroke", "scene": "plain", "paths": 1000,
         "tolerance": 0.1, "join": "miter", "cap": "butt", "bits": 16, "mode": "per_path"},
        # A large drawing: curve paths of log-normal length with round joins and caps and a width
        # of their own, all in one vertex buffer.
        {"name": "stroke drawing", "op": "batch", "kind": "stroke", "scene": "curves",
         "paths": 200000, "tolerance": 0.05, "join": "round", "cap": "round", "bits": 32,
         "mode": "global"},
        # A map layer: polylines, most of them a handful of points and a few very long, whose
        # joins are mixed.
        {"name": "stroke map", "op": "batch", "kind": "stroke", "scene": "polylines",
         "paths": 400001, "tolerance": 0.1, "join": "mixed", "cap": "butt", "bits": 32,
         "mode": "global"},
        # A shader-driven stroke (dashes, gradients along the line): every vertex with its normal,
        # side and distance along the path.
        {"name": "stroke with attributes", "op": "batch", "kind": "stroke", "scene": "curves",
         "paths": 20000, "tolerance": 0.1, "join": "bevel", "cap": "square", "bits": 32,
         "mode": "global", "vertices": "records"},
        # Pen input: a width per point (pressure).
        {"name": "stroke variable width", "op": "batch", "kind": "stroke", "scene": "curves",
         "paths": 10001, "tolerance": 0.1, "join": "round", "cap": "round", "bits": 32,
         "mode": "global", "vertices": "widths"},
        # Strokes that carry the user's own values per end point (a colour and a time), handed to
        # every vertex.
        {"name": "stroke custom values", "op": "batch", "kind": "stroke", "scene": "curves",
         "paths": 9999, "tolerance": 0.1, "join": "miter", "cap": "butt", "bits": 32,
         "mode": "global", "vertices": "custom"},
        # A page of text: a few hundred glyphs.
        {"name": "fill page", "op": "batch", "kind": "fill", "scene": "glyphs", "paths": 777,
         "tolerance": 0.1, "rule": "even_odd", "bits": 16, "mode": "per_path"},
        # A document, or a glyph atlas built in one go.
        {"name": "fill document", "op": "batch", "kind": "fill", "scene": "glyphs", "paths": 30000,
         "tolerance": 0.1, "rule": "non_zero", "bits": 32, "mode": "global"},
        # A drawing whose paths and results live in host memory (pinned), end to end.
        {"name": "stroke host buffers", "op": "host", "kind": "stroke", "scene": "curves",
         "paths": 10000, "tolerance": 0.05, "join": "round", "cap": "round", "bits": 32,
         "mode": "global"},
        # Flattening alone, for programs that walk or measure the polylines themselves.
        {"name": "flatten drawing", "op": "flatten", "kind": "flatten", "scene": "curves",
         "paths": 40000, "tolerance": 0.02},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    tol = round(math.exp(rng.uniform(math.log(0.02), math.log(0.5))), 4)
    join = rng.choice(sorted(JOINS))
    cap = rng.choice(sorted(CAPS))
    out = rng.choice([(16, "per_path"), (32, "per_path"), (32, "global")])
    seed = rng.randrange(1000)
    which = rng.randrange(9)
    if which == 0:
        return {"op": "path", "kind": "stroke", "segments": _log_int(rng, 1, 400),
                "scene_seed": seed, "tolerance": tol, "join": join, "cap": cap, "bits": 16}
    if which == 1:
        return {"op": "path", "kind": "fill", "scene_seed": seed, "tolerance": tol,
                "rule": rng.choice(sorted(RULES)), "bits": rng.choice([16, 32])}
    if which in (2, 3):
        scene = rng.choice(["plain", "curves"])
        return {"op": "batch", "kind": "stroke", "scene": scene,
                "scene_seed": seed, "paths": _log_int(rng, 2, 60000), "tolerance": tol,
                "join": join, "cap": cap, "bits": out[0], "mode": out[1]}
    if which == 4:
        return {"op": "batch", "kind": "stroke", "scene": "polylines",
                "scene_seed": seed, "paths": _log_int(rng, 3, 400000), "tolerance": tol,
                "join": "mixed", "cap": cap, "bits": out[0], "mode": out[1]}
    if which == 5:
        return {"op": "batch", "kind": "stroke", "scene": "curves",
                "scene_seed": seed, "paths": _log_int(rng, 2, 12000), "tolerance": tol,
                "join": join, "cap": cap, "bits": 32, "mode": out[1],
                "vertices": rng.choice(["records", "widths", "custom"])}
    if which in (6, 7):
        return {"op": "batch", "kind": "fill", "scene": "glyphs", "scene_seed": seed,
                "paths": _log_int(rng, 2, 30000), "tolerance": tol,
                "rule": rng.choice(sorted(RULES)), "bits": out[0], "mode": out[1]}
    return {"op": "flatten", "kind": "flatten", "scene": "curves", "scene_seed": seed,
            "paths": _log_int(rng, 1, 40000), "tolerance": tol}


# ---- inputs --------------------------------------------------------------------------------

def _scene(case, seed, paths=None):
    """The case's batch and option records (host arrays): its scene, turned by an angle and bent
    by a gentle wave that come from the seed, so that passes over other seeds differ in every
    coordinate and need about as much room for their outputs."""
    n = case.get("paths", 1) if paths is None else paths
    base = case.get("scene_seed", 7)
    scene = case.get("scene", "plain")
    if case["kind"] == "fill":
        batch, _ = workloads.glyph_fill(n, seed=base, fill_rule=RULES[case["rule"]])
        opts = np.zeros(1, FILL_OPTIONS_DTYPE)
        opts[0] = (case["tolerance"], RULES[case["rule"]], 0, 1)
        reach = 1024.0
    elif case["op"] == "path":
        rng = np.random.default_rng(base)
        batch = workloads._segment_paths(rng, np.array([case["segments"]]), rng.random(1) < 0.5)
        opts = np.zeros(1, STROKE_OPTIONS_DTYPE)
        opts["line_width"] = 4.0
        reach = 1024.0
    elif scene == "polylines":
        batch, opts = workloads.map_polylines(n, seed=base, tolerance=case["tolerance"])
        reach = 65536.0
    else:
        make = workloads.plain_stroke if scene == "plain" else workloads.batched_stroke
        batch, opts = make(n, seed=base)
        reach = 1024.0
    rng = np.random.default_rng(seed)
    angle, p, q = rng.uniform(0.0, 2.0 * math.pi, 3)
    x, y = (batch.points.reshape(-1, 2).astype(np.float64) - reach / 2).T
    x, y = (x * math.cos(angle) - y * math.sin(angle), x * math.sin(angle) + y * math.cos(angle))
    x, y = x + 3.0 * np.sin(y / 150.0 + p), y + 3.0 * np.sin(x / 150.0 + q)
    batch.points = (np.stack([x, y], axis=1) + reach / 2).astype(np.float32)
    if case["kind"] == "stroke":
        opts["tolerance"] = case["tolerance"]
        opts["miter_limit"] = 4.0
        opts["start_cap"] = opts["end_cap"] = CAPS[case["cap"]]
        if case["join"] != "mixed":
            opts["line_join"] = JOINS[case["join"]]
    return batch, opts


def _room(case):
    """(vertices, indices) that hold the outputs of any seed: the scene's flattened segments and
    a margin, for what joins, caps, arcs and crossings add."""
    sample = min(case.get("paths", 1), 2000)
    batch, _ = _scene(case, 1, sample)
    scale = 1.25 * case.get("paths", 1) / sample
    verbs = len(batch.verbs) * scale
    segments = float(_segment_counts(batch, case["tolerance"])[0].sum()) * scale
    if case["kind"] == "flatten":
        return int(segments + verbs) + 1024, 0
    vertices = int((segments if case["kind"] == "fill" else 2.0 * segments) + 20 * verbs) + 1024
    return vertices, 3 * vertices


def _tensor(shape, dtype, case, ctx):
    # What a pass does not write stays as it is here.
    if case["op"] in ("host", "path"):
        return torch.zeros(shape, dtype=dtype, pin_memory=case["op"] == "host")
    return torch.zeros(shape, dtype=dtype, device=f"cuda:{ctx.device}")


def prepare(case, seed):
    ctx = T.Context.default()
    batch, opts = _scene(case, seed)
    num_vertices, num_indices = _room(case)
    s = {"case": case, "ctx": ctx, "num_options": len(opts), "num_points": len(batch.points),
         "num_verbs": len(batch.verbs)}
    kind = case.get("vertices", "positions")
    # The program's own buffers, which take the outputs of scene after scene.
    out = s["out"] = {"vertices": _tensor((num_vertices, 6 if kind == "records" else 2),
                                          torch.float32, case, ctx)}
    if num_indices:
        out["indices"] = _tensor(num_indices, torch.int32 if case["bits"] == 32 else torch.int16,
                                 case, ctx)
    if case["op"] == "path":
        s["path"] = batch.path(0)
        if case["kind"] == "stroke":
            o = opts[0]
            s["options"] = StrokeOptions(int(o["start_cap"]), int(o["end_cap"]),
                                         int(o["line_join"]), float(o["line_width"]),
                                         float(o["miter_limit"]), float(o["tolerance"]))
            s["tessellator"] = T.StrokeTessellator(ctx)
        else:
            s["options"] = FillOptions(case["tolerance"], RULES[case["rule"]])
            s["tessellator"] = T.FillTessellator(ctx)
        s["out"] = {k: t.numpy() for k, t in out.items()}
        return s
    if case["op"] == "host":
        def pinned(a):
            t = torch.empty(a.nbytes, dtype=torch.uint8, pin_memory=True)
            t.numpy()[:] = np.ascontiguousarray(a).view(np.uint8).reshape(-1)
            return t
        s["in"] = [pinned(a) for a in (batch.verbs, batch.points, batch.verb_offsets,
                                       batch.point_offsets, opts)]
        s["batch"] = _native.CPathBatch(*[t.data_ptr() for t in s["in"][:4]], batch.num_paths)
        out["status"] = _tensor(batch.num_paths, torch.int32, case, ctx)
        return s
    s["batch"] = T.DeviceBatch.upload(batch, ctx.device)
    if case["op"] == "flatten":
        return s
    s["options"] = T.upload_options(opts, ctx.device)
    rng = np.random.default_rng(seed + 1)
    if kind == "widths":
        w = rng.uniform(0.5, 2.0, len(batch.points)).astype(np.float32)
        s["widths"] = torch.from_numpy(w).cuda(ctx.device)
    elif kind == "custom":
        a = rng.uniform(0.0, 1.0, (len(batch.points), 2)).astype(np.float32)
        s["custom"] = torch.from_numpy(a).cuda(ctx.device)
        out["source_ids"] = _tensor((num_vertices, 2), torch.int32, case, ctx)
        out["source_t"] = _tensor(num_vertices, torch.float32, case, ctx)
        out["custom"] = _tensor((num_vertices, 2), torch.float32, case, ctx)
    torch.cuda.synchronize()
    return s


def _mode(case):
    return T.INDEX_GLOBAL if case["mode"] == "global" else T.INDEX_PER_PATH


def _check(ctx, r):
    if r != T.LYON_OK:
        raise T.TessellationError(r, ctx.last_error())


def _view(ctx, ptr, shape, typestr):
    return torch.as_tensor(T._CudaArray(ptr, shape, typestr), device=f"cuda:{ctx.device}")


def run(s):
    case, ctx, out = s["case"], s["ctx"], s["out"]
    lib = ctx.lib
    if case["op"] == "path":
        # tessellate_path appends to the builder's buffers; the program copies them to its own.
        buffers = T.VertexBuffers(case["bits"])
        s["tessellator"].tessellate_path(s["path"], s["options"], T.BuffersBuilder(buffers))
        out["vertices"][:len(buffers.vertices)] = buffers.vertices
        out["indices"][:len(buffers.indices)] = buffers.indices.view(out["indices"].dtype)
        return {"vertices": out["vertices"], "indices": out["indices"],
                "counts": np.array([len(buffers.vertices), len(buffers.indices)])}
    nv, ni, failed = ctypes.c_uint64(), ctypes.c_uint64(), ctypes.c_uint32()
    if case["op"] == "host":
        _check(ctx, lib.lyon_gpu_stroke_paths_host(
            ctx.h, ctypes.byref(s["batch"]), s["in"][4].data_ptr(), s["num_options"],
            case["bits"], _mode(case), 0, out["vertices"].data_ptr(), out["vertices"].shape[0],
            out["indices"].data_ptr(), out["indices"].shape[0], out["status"].data_ptr(),
            ctypes.byref(nv), ctypes.byref(ni)))
        return dict(out, counts=np.array([nv.value, ni.value]))
    batch = s["batch"].c()
    if case["op"] == "flatten":
        pts, offs = ctypes.c_void_p(), ctypes.c_void_p()
        _check(ctx, lib.lyon_gpu_flatten_paths(ctx.h, ctypes.byref(batch), case["tolerance"],
                                               ctypes.byref(pts), ctypes.byref(offs),
                                               ctypes.byref(nv)))
        with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream)):
            out["vertices"][:nv.value] = _view(ctx, pts.value, (nv.value, 2), "<f4")
        return {"points": out["vertices"],
                "offsets": _view(ctx, offs.value, (s["num_verbs"] + 1,), "<i4")}
    if "vertices" not in case:
        # Sizes first, then straight into the program's own buffers.
        kind = 0 if case["kind"] == "stroke" else 1
        args = (ctx.h, kind, ctypes.byref(batch), s["options"].data_ptr(), s["num_options"],
                case["bits"], _mode(case), 0)
        _check(ctx, lib.lyon_gpu_query_sizes(*args, ctypes.byref(nv), ctypes.byref(ni),
                                             ctypes.byref(failed)))
        if nv.value > out["vertices"].shape[0] or ni.value > out["indices"].shape[0]:
            raise ValueError("the program's buffers are too small")
        res = _native.CBatchOutput()
        _check(ctx, lib.lyon_gpu_emit_into(*args, out["vertices"].data_ptr(),
                                           out["indices"].data_ptr(), ctypes.byref(res)))
        n = s["batch"].num_paths
        return dict(out, status=_view(ctx, res.status, (n,), "<i4"),
                    vertex_offsets=_view(ctx, res.vertex_offsets, (n + 1,), "<i8"),
                    index_offsets=_view(ctx, res.index_offsets, (n + 1,), "<i8"))
    kind = case["vertices"]
    res = T.tessellate_paths(case["kind"], s["batch"], s["options"], s["num_options"],
                             case["bits"], _mode(case), 0, ctx, attributes=kind == "records",
                             widths=s.get("widths"), custom_attributes=s.get("custom"))
    n, m = res.total_vertices, res.total_indices
    # The context's buffers are good until its next call: the program takes them over on the
    # context's own stream.
    with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream)):
        out["indices"][:m] = res.indices()
        if kind == "records":
            out["vertices"][:n] = res.records()
        else:
            out["vertices"][:n] = res.vertices()
        if kind == "custom":
            sources = res.sources()
            out["source_ids"][:n] = sources[:, :2]
            out["source_t"][:n] = sources.view(torch.float32)[:, 2]
            out["custom"][:n] = res.custom_attributes()
    vertex_offsets, index_offsets = res.offsets()
    outputs = dict(out, vertex_offsets=vertex_offsets, index_offsets=index_offsets,
                   status=res.statuses())
    if kind == "records":
        records = outputs.pop("vertices")
        outputs.update(vertices=records[:, :5], sides=records.view(torch.int32)[:, 5])
    return outputs


# ---- what a pass cannot do without -----------------------------------------------------------

def _segment_counts(batch, tolerance):
    """Flattened segments per verb (Wang's bound, in f32 with lyon's operations), each verb's
    first point and its kind."""
    verbs = batch.verbs
    step = np.array([1, 2, 3, 1, 1, 0])[verbs]
    first = np.cumsum(step) - step
    pts = np.asarray(batch.points, np.float32).reshape(-1, 2)
    tol = np.float32(tolerance)
    d = np.float32(1.0) / (np.float32(8.0) * tol)
    two, six = np.float32(2.0), np.float32(6.0)
    n = np.where((verbs == 0), 1, 0).astype(np.float32)

    def wang(err4):
        r = np.maximum(np.sqrt(np.sqrt(err4)), np.float32(1.0))
        small = np.searchsorted((np.arange(1, 25, dtype=np.float64) ** 4), err4) + 1
        return np.where(err4 <= 331776.0, small.astype(np.float32), r)

    def dot(v):
        return v[:, 0] * v[:, 0] + v[:, 1] * v[:, 1]

    q = np.nonzero(verbs == 1)[0]
    a, c, b = pts[first[q] - 1], pts[first[q]], pts[first[q] + 1]
    n[q] = wang(dot(((a - c * two) + b) * two) * d * d)
    q = np.nonzero(verbs == 2)[0]
    a, c, e, b = pts[first[q] - 1], pts[first[q]], pts[first[q] + 1], pts[first[q] + 2]
    n[q] = wang(np.maximum(dot(((a - c * two) + e) * six), dot(((c - e * two) + b) * six)) * d * d)
    return n, first


def work(case):
    # Counted on a sample of the scene: per flattened segment two vertices and six indices for a
    # stroke, one vertex and three indices for a fill, one point when flattening.
    paths = case.get("paths", 1)
    sample = min(paths, 2000)
    batch, opts = _scene(case, 12345, sample)
    scale = paths / sample
    segments = float(_segment_counts(batch, case["tolerance"])[0].astype(np.uint32).sum()) * scale
    inputs = (batch.verbs.nbytes + batch.points.nbytes + 8.0 * sample +
              (opts.nbytes if len(opts) > 1 else 0)) * scale
    if case["kind"] == "flatten":
        return {"bytes": inputs + 8.0 * segments + 4.0 * len(batch.verbs) * scale,
                "flops": 14.0 * segments}
    per_index = case["bits"] / 8
    offsets = 0.0 if case["op"] != "batch" else 20.0 * paths
    if case["kind"] == "fill":
        return {"bytes": inputs + offsets + segments * (8.0 + 3.0 * per_index),
                "flops": 40.0 * segments * math.log2(max(segments / paths, 2.0))}
    vertex = {"positions": 8.0, "records": 24.0, "widths": 8.0, "custom": 28.0}
    vertex = vertex[case.get("vertices", "positions")]
    return {"bytes": inputs + offsets + segments * (2.0 * vertex + 6.0 * per_index),
            "flops": 60.0 * segments}


# ---- the same outputs in 64 bits -------------------------------------------------------------

def exact(case, seed):
    # A tessellation has as many vertices as its decisions in f32 say (a bend that folds, a join's
    # arc split once more), so arithmetic in f64 gives another list and no value to hold a vertex
    # against; its indices and counts are whole numbers. Flattened points have one. Above 40,000
    # paths it takes too long.
    if case["op"] == "flatten" and case["paths"] <= 40000:
        points = _exact_flattening(case, seed)
        room = np.zeros((_room(case)[0], 2))
        room[:len(points)] = points
        return {"points": room, "offsets": None}
    return None


def _exact_flattening(case, seed):
    """Points at t = k / n of every curve, in f64."""
    batch, _ = _scene(case, seed)
    nf, first = _segment_counts(batch, case["tolerance"])
    n = nf.astype(np.int64)
    pts = batch.points.astype(np.float64)
    verb = np.repeat(np.arange(len(n)), n)
    k = np.arange(len(verb)) - np.repeat(np.cumsum(n) - n, n) + 1
    t = np.minimum(k / nf.astype(np.float64)[verb], 1.0)
    t[k == n[verb]] = 1.0
    out = np.empty((len(verb), 2))
    kind, f = batch.verbs[verb], first[verb]
    m = kind == 0
    out[m] = pts[f[m]]
    m = kind == 1
    u, v = t[m, None], 1.0 - t[m, None]
    out[m] = v * v * pts[f[m] - 1] + 2 * u * v * pts[f[m]] + u * u * pts[f[m] + 1]
    m = kind == 2
    u, v = t[m, None], 1.0 - t[m, None]
    out[m] = (v ** 3 * pts[f[m] - 1] + 3 * u * v * v * pts[f[m]] + 3 * u * u * v * pts[f[m] + 1] +
              u ** 3 * pts[f[m] + 2])
    return out
