"""Vertices inside a filled shape: the span on both sides of such a vertex is the same one, and
takes it twice. Compared with the oracle exactly."""

import numpy as np
import pytest

from lyon_gb300.options import FillRule, fill_options_array
from lyon_gb300.path import Path, PathBatch

pytestmark = pytest.mark.gpu

LINE, BEGIN, CLOSE = 0, 3, 4


def _nested(n, sides, seed):
    """A square and, inside it, n polygons of the same direction (windings of two and more)."""
    rng = np.random.default_rng(seed)
    polys = [np.array([(0, 0), (200, 1), (201, 200), (1, 199)], np.float64)]
    for _ in range(n):
        a = np.arange(sides) * (2 * np.pi / sides) + rng.uniform(0, 6)
        polys.append(rng.uniform(30, 170, 2) + rng.uniform(2, 25) * np.stack([np.cos(a), np.sin(a)], 1))
    verbs, points = [], []
    for p in polys:
        verbs += [BEGIN] + [LINE] * (len(p) - 1) + [CLOSE]
        points += list(p) + [p[0]]
    return Path(np.array(verbs, np.uint8), np.array(points, np.float32).reshape(-1, 2))


@pytest.mark.parametrize("orientation", [0, 1])
@pytest.mark.parametrize("n,sides", [(1, 3), (1, 40), (9, 5), (60, 7)])
def test_inner_vertices(n, sides, orientation):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gpu_helpers
    batch = PathBatch.from_paths([_nested(n, sides, s) for s in range(40)])
    opts = fill_options_array([(0.01, FillRule.NonZero, orientation, 1)])
    s = gpu_helpers.compare_per_path("fill", batch, opts, index_bits=32, rtol=0.0,
                                     allow_near_ties=False)
    assert not s["mismatches"], s["mismatches"][:10]
    assert np.array_equal(s["gpu"]["vertices"], s["oracle"]["vertices"])
