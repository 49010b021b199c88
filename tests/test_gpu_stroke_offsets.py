"""Strokes of batches whose verb offsets run backwards.

Such a batch is no partition of its verbs: the verb-parallel count leaves it to the walk of one
path by one warp, which takes every path by its own two offsets. The first call of a context
comes before anything has been written to the verbs' slots, so nothing there may be followed.
"""

import numpy as np
import pytest

import test_gpu_stroke_verbs as sv
from lyon_gb300 import tessellation as T
from lyon_gb300.path import PathBatch

pytestmark = pytest.mark.gpu


@pytest.fixture
def fresh():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    # Device memory handed out next holds no zeros.
    torch.full((64 << 20,), 255, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    c = T.Context(0)
    yield c
    c.close()


def backwards(form, n, seed):
    batch = sv.rough_paths(n, seed)
    vo, po = batch.verb_offsets.copy(), batch.point_offsets.copy()
    if form == "last":        # the last path ends before it starts
        vo, po = np.append(vo, vo[-1] - 1), np.append(po, po[-1])
    elif form == "first":     # so does the first one
        vo, po = np.append(vo[1], vo), np.append(po[1], po)
    elif form == "overlap":   # a path in the middle; its neighbours share verbs
        vo[n // 2], po[n // 2] = vo[n // 2 + 1], po[n // 2 + 1]
        vo[n // 2 + 1] -= 1
    elif form == "far":       # the batch ends before most of its paths
        vo[-1], po[-1] = vo[1], po[1]
    elif form == "reversed":  # every path
        vo, po = vo[::-1].copy(), po[::-1].copy()
    return PathBatch(batch.verbs, batch.points, vo, po)


FORMS = ["last", "first", "overlap", "far", "reversed"]


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("n", [2, 40, 3000])
def test_first_call_of_a_context(fresh, form, n):
    batch = backwards(form, n, 7 + n)
    sv.check(fresh, batch, sv.options(np.random.default_rng(n), batch.num_paths, tol=0.1))


@pytest.mark.parametrize("form", FORMS)
def test_after_a_larger_batch(fresh, form):
    rng = np.random.default_rng(3)
    good = sv.rough_paths(3000, 5)
    opts = sv.options(rng, good.num_paths, tol=0.1)
    small = backwards(form, 3, 6)
    for _ in range(2):  # slots of 3,000 paths, then a batch of few; and the large one again
        sv.check(fresh, good, opts)
        sv.check(fresh, small, sv.options(rng, small.num_paths, tol=0.1))
    sv.check(fresh, good, opts)


@pytest.mark.parametrize("how", sv.STEPPED)
@pytest.mark.parametrize("n", [1, 50])
def test_stepped_outputs_on_a_first_call(fresh, how, n):
    batch = sv.rough_paths(n, 20 + n)
    opts = sv.options(np.random.default_rng(n), n, tol=0.1)
    opts["line_width"] = np.maximum(opts["line_width"], 0.3)
    a = sv.stepped(fresh, batch, opts, how, by_path=True)
    sv.same_bits(a, sv.stepped(fresh, batch, opts, how))
