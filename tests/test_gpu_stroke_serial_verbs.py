"""Curves that the verb-parallel stroke would have one thread replay: short ones it does, long ones
and those whose skip test is not ruled out go to the walk of their path, 32 steps at a time."""

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


def curves(paths, per, scale, seed, turning=1.0, at=0.0):
    """Cubics; a share of them has its points on one line and turns round twice."""
    rng = np.random.default_rng(seed)
    verbs, pts, vo, po = [], [], [0], [0]
    for _ in range(paths):
        p = at + rng.uniform(0, 300, 2)
        verbs.append(Verb.BEGIN)
        pts.append(p)
        for _ in range(per):
            a = rng.uniform(0, 2 * np.pi)
            d = np.array([np.cos(a), np.sin(a)]) * scale * rng.uniform(0.5, 2)
            e = np.array([d[1], -d[0]])
            if rng.random() < turning:
                pts += [p + 4 * d, p - 3 * d, p + d]
            else:
                pts += [p + 0.3 * d + 0.2 * e, p + 0.7 * d - 0.2 * e, p + d]
            verbs.append(Verb.CUBIC_TO)
            p = p + d
        verbs.append(Verb.CLOSE if rng.random() < 0.5 else Verb.END)
        if verbs[-1] == Verb.CLOSE:
            pts.append(pts[po[-1]])
        vo.append(len(verbs))
        po.append(len(pts))
    return PathBatch(np.array(verbs, np.uint8), np.array(pts, np.float32).reshape(-1, 2),
                     np.array(vo, np.uint32), np.array(po, np.uint32))


# About 10 to 600 steps a curve, on both sides of the most a thread takes (35 for a path of one
# curve, 50 for one of ten).
@pytest.mark.parametrize("scale", [3.0, 20.0, 60.0, 150.0, 5000.0])
@pytest.mark.parametrize("paths,per,turning", [(1, 1, 1.0), (40, 10, 0.5), (400, 12, 0.1)])
def test_steps_of_a_thread(ctx, paths, per, turning, scale):
    batch = curves(paths, per, scale, 3, turning)
    sv.check(ctx, batch, sv.options(np.random.default_rng(4), batch.num_paths, tol=0.1))


@pytest.mark.parametrize("at", [0.0, 2e4, 1e6])
@pytest.mark.parametrize("width", [1.0, 400.0, 1e4])
def test_skips_that_are_not_ruled_out(ctx, width, at):
    # Short edges against the size of the coordinates and the width.
    batch = curves(60, 8, 30.0, 7, 0.2, at)
    o = sv.options(np.random.default_rng(4), batch.num_paths, tol=0.01)
    o["line_width"] = width
    sv.check(ctx, batch, o)
    for how in ("records", "widths", "sources"):
        sv.same_bits(sv.stepped(ctx, batch, o, how, by_path=True), sv.stepped(ctx, batch, o, how))


def test_one_long_curve_is_no_thread_s_work(ctx):
    # Against the same path by the walk alone (a last path whose offsets run backwards).
    batch = curves(1, 1, 1e4, 8)
    vo = np.append(batch.verb_offsets, batch.verb_offsets[-1] - 1)
    po = np.append(batch.point_offsets, batch.point_offsets[-1])
    walked = PathBatch(batch.verbs, batch.points, vo.astype(np.uint32), po.astype(np.uint32))
    opts = sv.options(np.random.default_rng(0), 1, tol=0.1, join=0)
    opts["line_width"] = 2.0
    od = T.upload_options(opts, 0)

    def best(b):
        db, times = T.DeviceBatch.upload(b, 0), []
        for _ in range(10):
            t = time.perf_counter()
            T.tessellate_paths("stroke", db, od, 1, 32, T.INDEX_GLOBAL, 0, ctx)
            ctx.synchronize()
            times.append(time.perf_counter() - t)
        return min(times)
    t, walk = best(batch), best(walked)
    print(t, walk)
    assert t < 2.5 * walk
