"""Flattening of a view from the middle of a batch: verbs before the view's first offset belong to
no path and have no points, whatever an earlier call left in the context's arrays."""

import ctypes

import numpy as np
import pytest

from lyon_gb300 import tessellation as T
from lyon_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    c = T.Context(0)
    yield c
    c.close()


def flatten(ctx, db, tolerance, num_verbs):
    import torch
    pts, offs, total = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_uint64()
    cb = db.c()
    r = ctx.lib.lyon_gpu_flatten_paths(ctx.h, ctypes.byref(cb), tolerance, ctypes.byref(pts),
                                       ctypes.byref(offs), ctypes.byref(total))
    assert r == T.LYON_OK, ctx.last_error()
    ctx.synchronize()

    def host(ptr, shape, kind):
        return torch.as_tensor(T._CudaArray(ptr, shape, kind), device="cuda").cpu().numpy().copy()
    return (host(pts.value, (total.value, 2), "<f4") if total.value else np.zeros((0, 2), np.float32),
            host(offs.value, (num_verbs + 1,), "<i4"))


@pytest.mark.parametrize("first,last", [(0, 40), (1, 40), (17, 23), (39, 40)])
def test_view_after_a_larger_batch(ctx, first, last):
    big, _ = workloads.batched_stroke(3000, seed=1)
    flatten(ctx, T.DeviceBatch.upload(big, 0), 0.05, len(big.verbs))
    batch, _ = workloads.batched_stroke(40, seed=2)
    db = T.DeviceBatch.upload(batch, 0)
    want, want_offsets = flatten(ctx, db, 0.05, len(batch.verbs))
    v0, v1 = int(batch.verb_offsets[first]), int(batch.verb_offsets[last])
    flatten(ctx, T.DeviceBatch.upload(big, 0), 0.05, len(big.verbs))
    db.verb_offsets = db.verb_offsets[first:last + 1]
    db.point_offsets = db.point_offsets[first:last + 1]
    db.num_paths = last - first
    points, offsets = flatten(ctx, db, 0.05, v1)
    assert not offsets[:v0 + 1].any()
    assert np.array_equal(offsets[v0:], want_offsets[v0:v1 + 1] - want_offsets[v0])
    assert np.array_equal(points, want[want_offsets[v0]:want_offsets[v1]])


def test_offsets_that_run_backwards(ctx):
    # The batch ends before its first path does: verbs past the end have no place in the outputs.
    batch, _ = workloads.batched_stroke(40, seed=3)
    db = T.DeviceBatch.upload(batch, 0)
    want, want_offsets = flatten(ctx, db, 0.05, len(batch.verbs))
    end = int(batch.verb_offsets[5])
    vo = np.array([0, batch.verb_offsets[30], end], np.int32)
    po = np.array([0, batch.point_offsets[30], batch.point_offsets[5]], np.int32)
    import torch
    db.verb_offsets, db.point_offsets = torch.from_numpy(vo).cuda(), torch.from_numpy(po).cuda()
    db.num_paths = 2
    torch.cuda.synchronize()
    points, offsets = flatten(ctx, db, 0.05, end)
    assert np.array_equal(offsets, want_offsets[:end + 1])
    assert np.array_equal(points, want[:want_offsets[end]])
