"""Where the verb-parallel stroke takes verbs and paths in groups: 32 lines at once in the sums along
a path, paths of more than 64 verbs by blocks unless they are lines, tiles that shrink with the batch.
Bit for bit against the walk and the thread per path."""

import numpy as np
import pytest

import test_gpu_stroke_verbs as sv
from lyon_gb300.path import PathBatch, Verb

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from lyon_gb300 import tessellation as T
    c = T.Context(0)
    yield c
    c.close()


def rows(lengths, seed):
    """One path per entry; an entry lists the rows of lines between curves and sub-path breaks."""
    rng = np.random.default_rng(seed)
    verbs, pts, vo, po = [], [], [0], [0]
    for path in lengths:
        p = rng.uniform(0, 400, 2)
        verbs.append(Verb.BEGIN)
        pts.append(p)
        for j, row in enumerate(path):
            for _ in range(row):
                p = p + rng.normal(0, 8, 2) * (rng.random() > 0.05)  # now and then a merge
                verbs.append(Verb.LINE_TO)
                pts.append(p)
            if j + 1 < len(path):
                if j % 2:
                    verbs += [Verb.END, Verb.BEGIN]
                    p = rng.uniform(0, 400, 2)
                    pts.append(p)
                else:
                    q = p + rng.normal(0, 15, (3, 2)).cumsum(0)
                    verbs.append(Verb.CUBIC_TO)
                    pts += list(q)
                    p = q[2]
        verbs.append(Verb.END)
        vo.append(len(verbs))
        po.append(len(pts))
    return PathBatch(np.array(verbs, np.uint8), np.array(pts, np.float32).reshape(-1, 2),
                     np.array(vo, np.uint32), np.array(po, np.uint32))


ROWS = [[1], [2], [31], [32], [33], [62], [63], [64], [65], [300], [1, 1, 1, 1], [30, 1, 33, 2],
        [0, 5, 0, 5], [32, 32, 32], [100, 100], [1000, 3], [3, 1000, 40, 40, 40], [0, 0, 0, 0, 0]]


@pytest.mark.parametrize("how", sv.STEPPED)
@pytest.mark.parametrize("times", [1, 40])
def test_rows_of_lines(ctx, how, times):
    batch = rows(ROWS * times, 3)
    o = sv.options(np.random.default_rng(4), batch.num_paths, tol=0.1)
    o["line_width"] = np.maximum(o["line_width"], 0.3)
    sv.same_bits(sv.stepped(ctx, batch, o, how, by_path=True), sv.stepped(ctx, batch, o, how))


# Verbs per tile: from the least (32 for the steppers, 128 for the tails) to the most (512 and 1024).
@pytest.mark.parametrize("n", [1, 40, 700, 6000, 60000])
def test_tiles(ctx, n):
    batch = rows([[2], [1], [3, 1]] * (n // 3 + 1), n)
    o = sv.options(np.random.default_rng(n), batch.num_paths, tol=0.1)
    o["line_width"] = np.maximum(o["line_width"], 0.3)
    sv.check(ctx, batch, o)
    for how in ("widths", "sources records"):
        sv.same_bits(sv.stepped(ctx, batch, o, how, by_path=True), sv.stepped(ctx, batch, o, how))


@pytest.mark.parametrize("how", ["records", "sources records"])
@pytest.mark.parametrize("n", [12288, 12289])
def test_sums_beside_the_count_or_after_it(ctx, how, n):
    batch = rows([[2, 3], [1], [40, 40]] * (n // 3) + [[1]] * (n % 3), n)
    o = sv.options(np.random.default_rng(n), batch.num_paths, tol=0.1)
    o["line_width"] = np.maximum(o["line_width"], 0.3)
    sv.same_bits(sv.stepped(ctx, batch, o, how, by_path=True), sv.stepped(ctx, batch, o, how))
