"""Attribute records of variable-width strokes with several sub-paths.

A sub-path's advancement starts where lyon's point buffer left off at the end of the one before
(stroke.rs:1359): with a variable width a skipped flattening step replaces a point of the buffer,
so that is no running sum over the kept points, and a closed sub-path may end with two points
left.
"""

import numpy as np
import pytest

import test_gpu_stroke_verbs as sv
from lyon_gb300 import tessellation as T
from lyon_gb300.options import STROKE_OPTIONS_DTYPE
from lyon_gb300.path import PathBatch, Verb
from oracle import lyon_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    c = T.Context(0)
    yield c
    c.close()


def batch_of(cubics, closed, tails=None):
    """Per path: Begin, a cubic, Close or End, then another sub-path of one line."""
    verbs, pts, vo, po = [], [], [0], [0]
    for k, q in enumerate(cubics):
        verbs += [Verb.BEGIN, Verb.CUBIC_TO, Verb.CLOSE if closed[k] else Verb.END,
                  Verb.BEGIN, Verb.LINE_TO, Verb.END]
        pts += list(q) + ([q[0]] if closed[k] else []) + [[5000, 0], [5100, 0]]
        vo.append(len(verbs))
        po.append(len(pts))
    return PathBatch(np.array(verbs, np.uint8), np.array(pts, np.float32).reshape(-1, 2),
                     np.array(vo, np.uint32), np.array(po, np.uint32))


def records(ctx, batch, opts, widths):
    import torch
    db, od = T.DeviceBatch.upload(batch, 0), T.upload_options(opts, 0)
    w = torch.from_numpy(widths).cuda()
    torch.cuda.synchronize()
    res = T.tessellate_paths("stroke", db, od, len(opts), 32, T.INDEX_PER_PATH, 0, ctx,
                             widths=w, attributes=True)
    ctx.synchronize()
    rec = res.records().cpu().numpy().view(T.STROKE_VERTEX_DTYPE).reshape(-1)
    return rec, res.offsets()[0].cpu().numpy(), res.statuses().cpu().numpy()


def test_start_of_the_second_sub_path(ctx):
    # The closed cubic leaves two points in lyon's buffer: the line starts at 15.1748, not at 0.
    batch = batch_of([[[0.47887674, -0.10222903], [-1.9204447, 1.3359492], [-5.766736, 7.6945114],
                       [-12.900506, 7.0578723]]], [True])
    opts = np.zeros(1, STROKE_OPTIONS_DTYPE)
    opts["line_width"], opts["tolerance"], opts["miter_limit"] = 20.0, 0.1957465, 4.0
    widths = np.array([1.98004377, 0.7200066, 1.2922924, 1.0477287, 1.5281104, 1.5469356,
                       1.6267770], np.float32)
    want = orc.batch("stroke", batch, opts, 32, 1, want_attributes=True, widths=widths)
    want = np.ascontiguousarray(want["attributes"][:, :3]).view(np.float32)[:, 2]
    rec, _, st = records(ctx, batch, opts, widths)
    assert st[0] == 0 and len(rec) == len(want)
    line = rec["x"] > 2500
    assert np.allclose(want[line].min(), 15.1748, rtol=0, atol=1e-3)
    assert np.array_equal(rec["advancement"], want)


@pytest.mark.parametrize("closed", [False, True])
def test_random_pairs_of_sub_paths(ctx, closed):
    rng = np.random.default_rng(17 + closed)
    n = 6000
    cubics = rng.normal(0, 6, (n, 4, 2)).cumsum(axis=1)
    batch = batch_of(cubics, [closed] * n)
    opts = np.zeros(n, STROKE_OPTIONS_DTYPE)
    opts["line_width"] = rng.uniform(2, 20, n)
    opts["tolerance"] = np.exp(rng.uniform(np.log(0.01), np.log(0.5), n))
    opts["miter_limit"] = 4.0
    opts["line_join"] = rng.choice([0, 2, 3], n)
    widths = rng.uniform(0.5, 2.0, len(batch.points)).astype(np.float32)
    want = orc.batch("stroke", batch, opts, 32, 8, want_attributes=True, widths=widths)
    rec, vo, st = records(ctx, batch, opts, widths)
    assert np.array_equal(st, want["status"])
    assert np.array_equal(vo, want["vtx_offsets"])
    adv = np.ascontiguousarray(want["attributes"][:, :3]).view(np.float32)[:, 2]
    line = rec["x"] > 2500  # the second sub-paths
    off = ~((rec["advancement"] == adv) | (np.isnan(rec["advancement"]) & np.isnan(adv)))
    assert not np.any(off & line), np.unique(np.searchsorted(vo, np.nonzero(off & line)[0],
                                                             "right") - 1).size


def test_rough_paths_of_several_sub_paths(ctx):
    # Against the thread that strokes a path as a whole.
    for seed in (61, 62, 63, 64):
        batch = sv.rough_paths(500, seed, max_verbs=6)
        o = sv.options(np.random.default_rng(seed), batch.num_paths)
        o["line_width"] = np.maximum(o["line_width"], 0.3)
        for how in ("widths records", "sources widths records"):
            sv.same_bits(sv.stepped(ctx, batch, o, how, by_path=True),
                         sv.stepped(ctx, batch, o, how))


def test_start_that_decides_a_fold(ctx):
    # A join's fold test takes differences of advancements, which round by their size: with another
    # start the third sub-path has one vertex more and a triangle less.
    verbs = [3, 0, 2, 4, 3, 0, 0, 2, 0, 0, 5, 3, 2, 2, 0, 1, 1, 0, 0, 4]
    pts = [[192.5571, 294.10443], [194.88756, 295.94342], [193.78716, 295.9947],
           [188.68097, 299.53302], [191.35272, 300.57715], [192.5571, 294.10443],
           [352.83078, 216.94138], [352.86792, 216.95052], [352.86792, 216.95052],
           [352.82217, 216.96696], [352.9137, 216.93405], [352.7754, 216.9609],
           [352.72232, 216.89346], [352.70685, 216.90799], [94.102104, 302.7594],
           [96.51862, 302.71045], [96.51862, 302.71045], [96.51862, 302.71045],
           [96.34326, 302.26913], [94.26125, 301.24524], [96.51751, 302.72067],
           [96.52352, 302.72314], [100.77119, 305.8152], [96.53413, 302.71524],
           [96.535545, 302.7136], [np.nan, np.nan], [96.544106, 302.72296],
           [96.53903, 302.7102], [94.102104, 302.7594]]
    widths = np.array([1.7532835, 1.8890697, 2.0728052, 0.6518197, 1.9705687, 1.525312, 0.84149075,
                       1.3264579, 2.372185, 1.4872794, 0.84606594, 0.6240128, 1.3036344, 2.102586,
                       1.0312787, 2.2327008, 1.5148836, 1.6129473, 2.3749108, 1.8366987, 1.8139644,
                       1.366115, 1.9680815, 2.2341533, 0.88740265, 1.7515548, 0.5827274, 0.7585378,
                       0.67546785], np.float32)
    batch = PathBatch(np.array(verbs, np.uint8), np.array(pts, np.float32),
                      np.array([0, len(verbs)], np.uint32), np.array([0, len(pts)], np.uint32))
    opts = np.zeros(1, STROKE_OPTIONS_DTYPE)
    opts["line_width"], opts["miter_limit"], opts["tolerance"] = 0.05, 1.0, 0.003
    import torch
    want = orc.batch("stroke", batch, opts, 32, 1, widths=widths)
    db, od = T.DeviceBatch.upload(batch, 0), T.upload_options(opts, 0)
    w = torch.from_numpy(widths).cuda()
    torch.cuda.synchronize()
    res = T.tessellate_paths("stroke", db, od, 1, 32, T.INDEX_GLOBAL, 0, ctx, widths=w)
    ctx.synchronize()
    assert (res.total_vertices, res.total_indices) == (309, 909)
    assert np.array_equal(res.indices().cpu().numpy().view(np.uint32), want["indices"])
    assert np.array_equal(res.vertices().cpu().numpy(), want["vertices"], equal_nan=True)
