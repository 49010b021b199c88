"""A stroke whose outputs fit the device's memory, but not beside the arrays that stroking verb by
verb takes, goes path by path."""

import ctypes

import numpy as np
import pytest

from lyon_gb300 import tessellation as T
from lyon_gb300.path import PathBatch, Verb

import test_gpu_stroke_verbs as sv

pytestmark = pytest.mark.gpu

N = 3_000_000  # lines: about 360 MB of verbs' arrays, 70 MB of vertices and 90 MB of indices


def test_outputs_before_the_verbs_arrays():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    per = 3000
    rng = np.random.default_rng(1)
    pts = rng.uniform(0, 500, (N // per, 1, 2)) + rng.normal(0, 5, (N // per, per, 2)).cumsum(1)
    verbs = np.tile(np.array([Verb.BEGIN] + [Verb.LINE_TO] * (per - 1) + [Verb.END], np.uint8),
                    N // per)
    batch = PathBatch(verbs, pts.reshape(-1, 2).astype(np.float32),
                      (np.arange(N // per + 1) * (per + 1)).astype(np.uint32),
                      (np.arange(N // per + 1) * per).astype(np.uint32))
    opts = sv.options(rng, 1, tol=0.1, join=0)
    db, od = T.DeviceBatch.upload(batch, 0), T.upload_options(opts, 0)
    c = T.Context(0)
    lib = c.lib
    try:
        res = T.tessellate_paths("stroke", db, od, 1, 32, T.INDEX_GLOBAL, 0, c)
        c.synchronize()
        want = res.vertices().clone(), res.indices().clone()
        out = res.total_vertices * 8 + res.total_indices * 4
    finally:
        c.close()
    torch.cuda.synchronize()
    held = []
    c = T.Context(0)
    try:
        # Room for the arrays (which a first call measures) and half the outputs.
        cb, nv, ni, nf = db.c(), ctypes.c_uint64(), ctypes.c_uint64(), ctypes.c_uint32()
        free0 = torch.cuda.mem_get_info()[0]
        assert lib.lyon_gpu_query_sizes(c.h, 0, ctypes.byref(cb), od.data_ptr(), 1, 32,
                                        T.INDEX_GLOBAL, 0, ctypes.byref(nv), ctypes.byref(ni),
                                        ctypes.byref(nf)) == T.LYON_OK
        arrays = free0 - torch.cuda.mem_get_info()[0]
        assert arrays > 2 * out, (arrays, out)
        # (In blocks: what the allocator rounds up stays small.)
        left = torch.cuda.mem_get_info()[0] - out // 2
        while left > 0:
            n = min(left, 32 << 30)
            held.append(torch.empty(n, dtype=torch.uint8, device="cuda"))
            left -= n
        res = T.tessellate_paths("stroke", db, od, 1, 32, T.INDEX_GLOBAL, 0, c)
        c.synchronize()
        assert torch.equal(res.vertices(), want[0]) and torch.equal(res.indices(), want[1])
    finally:
        held.clear()
        torch.cuda.empty_cache()
        c.close()
