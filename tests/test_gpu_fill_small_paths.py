"""Batches of many small paths on both sides of the rule that gives the simple ones to a thread each
and the others to a warp: sizes around 128, two to five peaks, curves, both orientations. Compared
with the oracle exactly."""

import numpy as np
import pytest

from lyon_gb300.options import FillRule, fill_options_array
from lyon_gb300.path import Path, PathBatch

pytestmark = pytest.mark.gpu

LINE, CUBIC, BEGIN, CLOSE, END = 0, 2, 3, 4, 5


def _ring(points, close=True):
    verbs = [BEGIN] + [LINE] * (len(points) - 1) + [CLOSE if close else END]
    pts = list(points) + ([points[0]] if close else [])
    return Path(np.array(verbs, np.uint8), np.array(pts, np.float32).reshape(-1, 2))


def _convex(n, rng):
    a = np.arange(n) * (2 * np.pi / n) + rng.uniform(0, 6)
    return _ring(rng.uniform(20, 80, 2) + rng.uniform(3, 20) * np.stack([np.cos(a), np.sin(a)], 1))


def _peaks(n, rng):
    """A comb of n teeth, one of them a little below the others."""
    x = np.arange(2 * n + 1)
    y = np.where(x % 2, 0.0, 10.0 + 0.1 * (x % 5))
    p = np.concatenate([np.stack([x, y], 1), [[2 * n + 1, 20.0], [-1.0, 21.0]]])
    return _ring(p * rng.uniform(0.5, 2) + rng.uniform(0, 50, 2), rng.random() < 0.8)


def _outline(n, size, rng):
    a = np.arange(3 * n) * (2 * np.pi / (3 * n)) + rng.uniform(0, 6)
    r = size * (1 + 0.3 * (np.arange(3 * n) % 3 == 1))
    p = rng.uniform(20, 80, 2) + r[:, None] * np.stack([np.cos(a), np.sin(a)], 1)
    p = np.concatenate([p, p[:1], p[:1]])
    return Path(np.array([BEGIN] + [CUBIC] * n + [CLOSE], np.uint8), p.astype(np.float32))


def _simple(i, rng):
    kind = i % 4
    if kind == 0:
        return _convex(3 + i % 9, rng)
    if kind == 1:
        return _outline(2, rng.uniform(1, 5), rng)
    if kind == 2:
        return _ring(rng.integers(0, 12, (2 + i % 3, 2)) * 1.25)
    return _peaks(1, rng)


def _others(rng):
    out = [_convex(n, rng) for n in (100, 125, 126, 127, 128, 300)]
    out += [_peaks(n, rng) for n in (2, 3, 4, 5, 30)]
    out += [_outline(n, s, rng) for n in (4, 8) for s in (3.0, 40.0, 400.0)]
    out += [_ring(rng.uniform(0, 50, (n, 2))) for n in (6, 9, 20)]
    out.append(Path(np.array([BEGIN, LINE, 9], np.uint8), np.zeros((3, 2), np.float32)))
    out.append(_ring([(0.0, 0.0), (5.0, float("nan")), (9.0, 3.0)]))
    out.append(_ring([(1.0, 1.0)]))
    return out


@pytest.mark.parametrize("orientation", [0, 1])
@pytest.mark.parametrize("simple", [12287, 12288, 24560])
def test_small_paths(simple, orientation):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gpu_helpers
    rng = np.random.default_rng(simple)
    kinds = [_simple(i, rng) for i in range(512)]
    paths = [kinds[i % 512] for i in range(simple)]
    for _ in range(1 if simple < 24560 else 20):  # the last is past 24,576 paths
        paths += _others(rng)
    paths = [paths[i] for i in rng.permutation(len(paths))]
    batch = PathBatch.from_paths(paths)
    opts = fill_options_array([(0.05, FillRule.NonZero, orientation, 1)])
    s = gpu_helpers.compare_per_path("fill", batch, opts, index_bits=32, rtol=0.0,
                                     allow_near_ties=False)
    assert not s["mismatches"], s["mismatches"][:10]
    assert np.array_equal(s["gpu"]["vertices"], s["oracle"]["vertices"], equal_nan=True)


@pytest.mark.parametrize("others", [13000, 13600])
def test_small_paths_among_as_many_others(others):
    # Threads sweep them while they are half of the batch.
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gpu_helpers
    rng = np.random.default_rng(others)
    kinds, comb = [_simple(i, rng) for i in range(256)], _peaks(5, rng)
    paths = [kinds[i % 256] for i in range(13300)] + [comb] * others
    paths = [paths[i] for i in rng.permutation(len(paths))]
    batch = PathBatch.from_paths(paths)
    opts = fill_options_array([(0.05, FillRule.EvenOdd, 0, 1)])
    s = gpu_helpers.compare_per_path("fill", batch, opts, index_bits=32, rtol=0.0,
                                     allow_near_ties=False)
    assert not s["mismatches"], s["mismatches"][:10]
    assert np.array_equal(s["gpu"]["vertices"], s["oracle"]["vertices"])


def test_sources_of_small_paths():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import gpu_helpers
    import test_gpu_fill_custom as custom
    rng = np.random.default_rng(8)
    kinds = [_simple(i, rng) for i in range(256)]
    paths = [kinds[i % 256] for i in range(12400)] + _others(rng)
    paths = [paths[i] for i in rng.permutation(len(paths))]
    batch = PathBatch.from_paths(paths)
    opts = fill_options_array([(0.05, FillRule.NonZero, 0, 1)])
    attrs = rng.uniform(0, 1, (len(batch.points), 2)).astype(np.float32)
    bad, _ = custom.compare_fill_custom(gpu_helpers, batch, opts, attrs)
    assert not bad, bad[:10]


def test_time_of_many_simple_paths():
    # 30,000 polygons of 32 points: a thread each takes less time than a warp each would, which is
    # what the same batch takes in three calls of 10,000.
    import time
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from lyon_gb300 import tessellation as T
    rng = np.random.default_rng(5)
    ring = [_convex(32, rng) for _ in range(200)]
    opts = T.upload_options(fill_options_array([(0.1, FillRule.NonZero, 0, 1)]), 0)
    c = T.Context(0)
    try:
        def best(n):
            db = T.DeviceBatch.upload(PathBatch.from_paths([ring[i % 200] for i in range(n)]), 0)
            times = []
            for _ in range(8):
                t = time.perf_counter()
                T.tessellate_paths("fill", db, opts, 1, 32, T.INDEX_GLOBAL, 0, c)
                c.synchronize()
                times.append(time.perf_counter() - t)
            return min(times)
        whole, third = best(30000), best(10000)
        print(whole, third)
        assert whole < 2.2 * third
    finally:
        c.close()
