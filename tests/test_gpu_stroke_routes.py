"""Batches on both sides of the rule that strokes many short paths path by path and others verb by
verb: bit for bit the same, and not much slower than the other way."""

import time

import numpy as np
import pytest

import test_gpu_stroke_verbs as sv
from lyon_gb300 import tessellation as T
from lyon_gb300.path import PathBatch, Verb

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    c = T.Context(0)
    yield c
    c.close()


def lines(n, points, seed, closed=False, long_one=0):
    """n polylines of `points` points (and one of `long_one`)."""
    rng = np.random.default_rng(seed)
    m = points + closed
    p = rng.uniform(0, 500, (n, 1, 2)) + rng.normal(0, 8, (n, points, 2)).cumsum(1)
    p[rng.random((n, points)) < 0.03] = p[0, 0]
    if closed:
        p = np.concatenate([p, p[:, :1]], axis=1)
    v = np.array([Verb.BEGIN] + [Verb.LINE_TO] * (points - 1)
                 + [Verb.CLOSE if closed else Verb.END], np.uint8)
    verbs, pts = np.tile(v, n), p.reshape(-1, 2)
    vo, po = np.arange(n + 1) * (points + 1), np.arange(n + 1) * m
    if long_one:
        verbs = np.concatenate([verbs, [Verb.BEGIN], [Verb.LINE_TO] * (long_one - 1), [Verb.END]])
        pts = np.concatenate([pts, rng.uniform(0, 500, (long_one, 2))])
        vo, po = np.append(vo, len(verbs)), np.append(po, len(pts))
    return PathBatch(verbs.astype(np.uint8), pts.astype(np.float32), vo.astype(np.uint32),
                     po.astype(np.uint32))


def cubics(n, per, seed):
    rng = np.random.default_rng(seed)
    p = rng.uniform(0, 500, (n, 1, 2)) + rng.normal(0, 15, (n, 3 * per + 1, 2)).cumsum(1)
    v = np.array([Verb.BEGIN] + [Verb.CUBIC_TO] * per + [Verb.END], np.uint8)
    return PathBatch(np.tile(v, n), p.reshape(-1, 2).astype(np.float32),
                     (np.arange(n + 1) * (per + 2)).astype(np.uint32),
                     (np.arange(n + 1) * (3 * per + 1)).astype(np.uint32))


def opts_for(batch, seed=1):
    o = sv.options(np.random.default_rng(seed), batch.num_paths, tol=0.1)
    o["line_width"] = np.maximum(o["line_width"], 0.3)
    return o


@pytest.mark.parametrize("n", [32767, 32768, 40000])
@pytest.mark.parametrize("points,closed,long_one", [(2, False, 0), (4, True, 0), (8, False, 0),
                                                    (9, False, 0), (3, False, 33), (3, False, 32)])
def test_short_lines(ctx, n, points, closed, long_one):
    batch = lines(n, points, n + points, closed, long_one)
    sv.check(ctx, batch, opts_for(batch))


@pytest.mark.parametrize("how", ["records", "sources", "sources records"])
@pytest.mark.parametrize("n,points", [(16383, 3), (16384, 3), (30000, 3), (30000, 12), (25000, 40)])
def test_records_and_sources_of_lines(ctx, how, n, points):
    batch = lines(n, points, n + points)
    o = opts_for(batch)
    sv.same_bits(sv.stepped(ctx, batch, o, how, by_path=True), sv.stepped(ctx, batch, o, how))


@pytest.mark.parametrize("how", ["widths", "widths records", "sources widths"])
@pytest.mark.parametrize("n,per", [(1, 2), (1, 30), (100, 3), (100, 12), (3000, 6), (20000, 20)])
def test_widths_of_lines_and_curves(ctx, how, n, per):
    for batch in (lines(n, per, n + per), cubics(n, max(1, per // 4), n)):
        o = opts_for(batch)
        sv.same_bits(sv.stepped(ctx, batch, o, how, by_path=True), sv.stepped(ctx, batch, o, how))


def test_single_paths_of_variable_width(ctx):
    # The shape of a path that comes in host arrays is known without asking the device.
    from lyon_gb300.options import StrokeOptions
    from lyon_gb300.path import Path
    from oracle import lyon_oracle as orc
    rng = np.random.default_rng(3)
    for k in (2, 3, 5, 9, 40):
        verbs = np.array([Verb.BEGIN] + [Verb.LINE_TO] * (k - 1) + [Verb.END], np.uint8)
        path = Path(verbs, rng.uniform(0, 100, (k, 2)).astype(np.float32))
        w = rng.uniform(0.5, 2, k).astype(np.float32)
        ref = orc.stroke(path, StrokeOptions(line_width=3.0), 16, widths=w)
        out = T.VertexBuffers(16)
        T.StrokeTessellator(ctx).tessellate_path(path, StrokeOptions(line_width=3.0),
                                                 T.BuffersBuilder(out), widths=w)
        assert np.array_equal(out.indices, ref.indices)
        assert np.array_equal(out.vertices, ref.vertices)


@pytest.mark.parametrize("how", ["positions", "records", "sources", "widths"])
def test_time_of_many_short_lines(ctx, how):
    # Against the same batch with a last path whose offsets run backwards, which goes path by path
    # whatever the rule says (after a first look at it that is part of the time).
    import torch
    batch = lines(200000, 3, 9)
    vo = np.append(batch.verb_offsets, batch.verb_offsets[-1] - 1).astype(np.uint32)
    po = np.append(batch.point_offsets, batch.point_offsets[-1]).astype(np.uint32)
    od = T.upload_options(opts_for(batch)[:1], 0)
    rng = np.random.default_rng(1)
    w = torch.from_numpy(rng.uniform(0.5, 2, len(batch.points)).astype(np.float32)).cuda()
    kw = {"positions": {}, "records": dict(attributes=True), "widths": dict(widths=w),
          "sources": dict(custom_attributes=w.reshape(-1, 1))}[how]
    torch.cuda.synchronize()

    def best(b):
        db, times = T.DeviceBatch.upload(b, 0), []
        for _ in range(8):
            t = time.perf_counter()
            T.tessellate_paths("stroke", db, od, 1, 32, T.INDEX_GLOBAL, 0, ctx, **kw)
            ctx.synchronize()
            times.append(time.perf_counter() - t)
        return min(times)
    t, path = best(batch), best(PathBatch(batch.verbs, batch.points, vo, po))
    print(how, t, path)
    assert t < 1.25 * path


def test_a_large_batch_after_a_small_one(ctx):
    # A context that has room for the large batch does not know its size beforehand.
    large, small = lines(2000, 500, 4), lines(1, 2, 5)
    od = T.upload_options(opts_for(large)[:1], 0)
    dl, ds = T.DeviceBatch.upload(large, 0), T.DeviceBatch.upload(small, 0)

    def call(db):
        t = time.perf_counter()
        res = T.tessellate_paths("stroke", db, od, 1, 32, T.INDEX_GLOBAL, 0, ctx)
        ctx.synchronize()
        return time.perf_counter() - t, res
    call(dl)
    again = min(call(dl)[0] for _ in range(5))
    want = call(dl)[1].vertices().clone()
    after = []
    for _ in range(5):
        call(ds)
        t, res = call(dl)
        after.append(t)
    assert bool((res.vertices() == want).all())
    print(again, after)
    assert min(after) < 2 * again


@pytest.mark.parametrize("how", ["positions", "records"])
def test_settings_of_the_path_by_path_stroke(ctx, how):
    # Short line-only paths by a thread each, long ones first, one block per SM: the same outputs,
    # and those of the walk by one warp. (A last path whose offsets run backwards sends all of them
    # path by path.)
    import ctypes
    from lyon_gb300 import _native
    batch = sv.rough_paths(800, 9)
    short = lines(700, 5, 3)
    verbs = np.concatenate([batch.verbs, short.verbs])
    pts = np.concatenate([batch.points, short.points])
    vo = np.concatenate([batch.verb_offsets, short.verb_offsets[1:] + batch.verb_offsets[-1]])
    po = np.concatenate([batch.point_offsets, short.point_offsets[1:] + batch.point_offsets[-1]])
    vo, po = np.append(vo, vo[-1] - 1), np.append(po, po[-1])
    b = PathBatch(verbs, pts, vo.astype(np.uint32), po.astype(np.uint32))
    o = opts_for(b)
    saved = _native.CStrokeTuning()
    ctx.lib.lyon_gpu_get_stroke_tuning(ctx.h, ctypes.byref(saved))
    out = []
    try:
        for tuning in ((0, 0, 0), (1024, 0, 32), (16, 1, 64), (0, 2, 5)):
            t = _native.CStrokeTuning(*tuning)
            assert ctx.lib.lyon_gpu_set_stroke_tuning(ctx.h, ctypes.byref(t)) == T.LYON_OK
            if how == "positions":
                sv.check(ctx, b, o)
            out.append(sv.stepped(ctx, b, o, "records" if how == "records" else "widths"))
    finally:
        ctx.lib.lyon_gpu_set_stroke_tuning(ctx.h, ctypes.byref(saved))
    for x in out[1:]:
        sv.same_bits(out[0], x)
