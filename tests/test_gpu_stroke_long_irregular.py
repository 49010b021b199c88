"""Long sub-paths of verbs that the steppers cannot start in the middle of: the steps before a
verb, which give the stepper its state, go back over a few verbs and not to the sub-path's start."""

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


def back_and_forth(paths, curves, seed, mixed=False):
    """Cubics whose points lie on one line and turn round twice; with `mixed` other verbs among
    them, some of whose end points merge with the step before."""
    rng = np.random.default_rng(seed)
    verbs, pts, vo, po = [], [], [0], [0]
    for _ in range(paths):
        p = rng.uniform(0, 300, 2)
        verbs.append(Verb.BEGIN)
        pts.append(p)
        for _ in range(curves):
            a = rng.uniform(0, 2 * np.pi)
            d = np.array([np.cos(a), np.sin(a)]) * rng.uniform(15, 60)
            kind = rng.integers(0, 6) if mixed else 5
            if kind == 0:
                verbs.append(Verb.LINE_TO)
                pts.append(p + d)
            elif kind == 1:    # ends in a short step
                verbs.append(Verb.CUBIC_TO)
                pts += [p + d * 2, p + d * (1 + 1e-6), p + d]
            elif kind == 2:
                verbs.append(Verb.QUADRATIC_TO)
                pts += [p + 0.5 * d + d[::-1], p + d]
            else:
                verbs.append(Verb.CUBIC_TO)
                pts += [p + 4 * d, p - 3 * d, p + d]
            p = p + d
        verbs.append(Verb.END)
        vo.append(len(verbs))
        po.append(len(pts))
    return PathBatch(np.array(verbs, np.uint8), np.array(pts, np.float32).reshape(-1, 2),
                     np.array(vo, np.uint32), np.array(po, np.uint32))


def plain(n, width=2.0):
    o = sv.options(np.random.default_rng(0), n, tol=0.1, join=0)
    o["line_width"], o["miter_limit"] = width, 4.0
    o["start_cap"] = o["end_cap"] = 0
    return o


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("how", sv.STEPPED)
def test_outputs(ctx, how, mixed):
    batch = back_and_forth(30, 60, 5, mixed)
    sv.same_bits(sv.stepped(ctx, batch, plain(1), how, by_path=True),
                 sv.stepped(ctx, batch, plain(1), how))


def test_time_is_not_that_of_all_verbs_before(ctx):
    # Records and vertex sources need the same sums along the path; the sources step every verb
    # besides, which takes many times that when each steps all verbs before it too.
    import torch
    batch = back_and_forth(1, 3000, 6)
    db, od = T.DeviceBatch.upload(batch, 0), T.upload_options(plain(1), 0)
    attrs = torch.ones((len(batch.points), 1), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()

    def best(**kw):
        times = []
        for _ in range(4):
            t = time.perf_counter()
            T.tessellate_paths("stroke", db, od, 1, 32, T.INDEX_GLOBAL, 0, ctx, **kw)
            ctx.synchronize()
            times.append(time.perf_counter() - t)
        return min(times)
    records, sources = best(attributes=True), best(custom_attributes=attrs)
    print(records, sources)
    assert sources < 2 * records
