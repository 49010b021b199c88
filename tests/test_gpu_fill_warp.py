"""The sweep of a warp per path at the sizes where its parts change: 32 active edges per ballot and
64 in shared memory, 8 pending edges, 32 spans, runs of 32 sorted events, 32 points of a curve, and
windings beyond one; and the batch sizes around which tiny paths go to a thread each. Compared with
the oracle exactly: vertices, indices and statuses.
"""

import numpy as np
import pytest

from lyon_gb300.options import FillRule, fill_options_array
from lyon_gb300.path import Path, PathBatch

pytestmark = pytest.mark.gpu

LINE, QUAD, BEGIN, CLOSE = 0, 1, 3, 4


def _polygons(*polygons):
    verbs, points = [], []
    for poly in polygons:
        verbs += [BEGIN] + [LINE] * (len(poly) - 1) + [CLOSE]
        points += list(poly) + [poly[0]]
    return Path(np.array(verbs, np.uint8), np.array(points, np.float32).reshape(-1, 2))


def _comb(teeth, up):
    """2 * teeth edges are active at once; a span per tooth on one side of the back."""
    pts = [(0.0, 100.0), (2.0 * teeth + 1.0, 100.0 + 0.3 * teeth)]
    for i in reversed(range(teeth)):
        pts += [(2.0 * i + 1.9, 90.0 + 0.01 * i), (2.0 * i + 1.0, 3.0 + 0.7 * (i % 5)),
                (2.0 * i + 0.3, 91.0 - 0.01 * i)]
    if not up:
        pts = [(x, -y) for x, y in pts]
    return pts


def _round(n, r=40.0, cx=0.0, cy=0.0):
    a = np.arange(n) * (2.0 * np.pi / n) + 0.1
    return [(float(cx + r * np.cos(t)), float(cy + r * np.sin(t))) for t in a]


def _fan(k):
    """k triangles that meet at one point: 2 * k edges begin there, and as many end."""
    fans = []
    for i in range(k):
        a, b = (2 * i - k) / k, (2 * i + 1 - k) / k
        fans.append([(0.0, 0.0), (50.0 * a, 40.0 + i), (50.0 * b, 40.0 + i)])
        fans.append([(0.0, 0.0), (50.0 * a, -40.0 - i), (50.0 * b, -40.0 - i)])
    return fans


def _bow(scale):
    return Path(np.array([BEGIN, QUAD, QUAD, CLOSE], np.uint8),
                np.array([(0, 0), (scale, 0.3 * scale), (0.1 * scale, scale),
                          (-scale, 0.6 * scale), (0, 0), (0, 0)], np.float32))


def _paths():
    out = [_polygons(_round(n)) for n in (3, 4, 15, 16, 31, 32, 33, 63, 64, 65, 127, 129, 300)]
    for teeth in (15, 16, 17, 31, 32, 33, 40):
        for up in (False, True):
            comb = _comb(teeth, up)
            y = 50.0 if up else -50.0
            band = [(-3.0, y), (2.0 * teeth + 3.0, y + 4.0), (2.0 * teeth + 3.0, y + 9.0),
                    (-3.0, y + 5.0)]
            out += [_polygons(comb), _polygons(comb, band)]
    out += [_polygons(*_fan(k)) for k in (1, 3, 4, 5, 16, 17, 40)]
    for times in (2, 3, 5):  # windings of `times`
        out.append(_polygons(*([_round(20)] * times), *([_round(7, 15.0, 3.0, 2.0)] * (times - 1))))
    # The number of steps grows with the square root of a curve's size: about 20 to 300 points.
    for steps in (1, 31, 32, 33, 63, 64, 65, 97):
        out.append(_bow(0.0125 * steps * steps))
    out.append(_polygons([(0.0, 0.0), (5.0, float("nan")), (9.0, 3.0), (1.0, 8.0)]))
    out.append(_polygons([(2.0, 2.0)], [(1.0, 1.0), (1.0, 1.0)]))
    return out


@pytest.mark.parametrize("orientation", [0, 1])
@pytest.mark.parametrize("rule", [FillRule.NonZero, FillRule.EvenOdd])
def test_sizes_of_the_warps_sweep(rule, orientation):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gpu_helpers
    paths = _paths()
    batch = PathBatch.from_paths(paths)
    opts = fill_options_array([(0.01, rule, orientation, 1)])
    s = gpu_helpers.compare_per_path("fill", batch, opts, index_bits=32, rtol=0.0,
                                     allow_near_ties=False)
    assert not s["mismatches"], s["mismatches"][:10]
    assert np.array_equal(s["gpu"]["vertices"], s["oracle"]["vertices"])


@pytest.mark.parametrize("tiny", [16383, 16384])
def test_tiny_paths_by_threads_among_others(tiny):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gpu_helpers
    rng = np.random.default_rng(tiny)
    # Up to 7 points (the closing one included), crossing itself as it comes; then larger ones,
    # small ones with a curve, and one verb list that no path may have.
    paths = [_polygons(list(map(tuple, rng.integers(0, 12, (2 + i % 5, 2)) * 1.25)))
             for i in range(tiny)]
    paths += [_polygons(_round(n)) for n in (7, 8, 33)] * 20 + [_bow(3.0)] * 20
    paths.insert(100, Path(np.array([BEGIN, LINE, 9], np.uint8), np.zeros((3, 2), np.float32)))
    paths = [paths[i] for i in rng.permutation(len(paths))]
    batch = PathBatch.from_paths(paths)
    opts = fill_options_array([(0.01, FillRule.EvenOdd, 0, 1)])
    s = gpu_helpers.compare_per_path("fill", batch, opts, index_bits=32, rtol=0.0,
                                     allow_near_ties=False)
    assert not s["mismatches"], s["mismatches"][:10]
    assert np.array_equal(s["gpu"]["vertices"], s["oracle"]["vertices"])
