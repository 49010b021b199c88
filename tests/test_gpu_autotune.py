"""The autotuners time the kernels that their settings are for, and keep no setting that the sample
says nothing about."""

import ctypes

import numpy as np
import pytest

import test_gpu_stroke_routes as routes
from lyon_gb300 import _native, workloads
from lyon_gb300 import tessellation as T

pytestmark = pytest.mark.gpu


@pytest.fixture
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    c = T.Context(0)
    yield c
    c.close()


def test_stroke_settings_are_timed_path_by_path(ctx):
    # One polyline of 40,000 points: a warp's walk of it takes milliseconds, verb by verb it is over
    # in a fraction of one.
    batch = routes.lines(10, 3, 1, long_one=40000)
    opts = routes.opts_for(batch)
    db, od = T.DeviceBatch.upload(batch, 0), T.upload_options(opts, 0)
    best, nc, times = _native.CStrokeTuning(), ctypes.c_uint32(), (ctypes.c_float * 16)()
    cb = db.c()
    before = T.tessellate_paths("stroke", db, od, len(opts), 32, T.INDEX_GLOBAL, 0, ctx)
    ctx.synchronize()
    ctx.lib.lyon_gpu_set_timing(ctx.h, 1)
    T.tessellate_paths("stroke", db, od, len(opts), 32, T.INDEX_GLOBAL, 0, ctx)
    ms = (ctypes.c_float * 4)()
    ctx.lib.lyon_gpu_last_timings(ctx.h, ms)
    ctx.lib.lyon_gpu_set_timing(ctx.h, 0)
    v = before.vertices().cpu().numpy()
    r = ctx.lib.lyon_gpu_autotune_stroke(ctx.h, ctypes.byref(cb), od.data_ptr(), len(opts), 0,
                                         ctypes.byref(best), times, ctypes.byref(nc))
    assert r == T.LYON_OK and nc.value == 16
    print(ms[3], list(times))
    assert min(times) > 4 * ms[3]
    # Later calls go verb by verb again.
    res = T.tessellate_paths("stroke", db, od, len(opts), 32, T.INDEX_GLOBAL, 0, ctx)
    ctx.synchronize()
    assert np.array_equal(res.vertices().cpu().numpy(), v)
    ctx.lib.lyon_gpu_set_timing(ctx.h, 1)
    T.tessellate_paths("stroke", db, od, len(opts), 32, T.INDEX_GLOBAL, 0, ctx)
    ctx.lib.lyon_gpu_last_timings(ctx.h, ms)
    assert ms[3] < min(times) / 2


@pytest.mark.parametrize("threads", [False, True])
def test_fill_keeps_the_number_of_threads_only_where_it_matters(ctx, threads):
    if threads:
        batch, opts = routes.lines(20000, 4, 2, closed=True), None
    else:
        batch, opts = workloads.glyph_fill(300, seed=47)
    if opts is None:
        opts = workloads.glyph_fill(1, seed=1)[1][:1]
    db, od = T.DeviceBatch.upload(batch, 0), T.upload_options(opts, 0)
    best, now, nc = _native.CFillTuning(), _native.CFillTuning(), ctypes.c_uint32()
    times = (ctypes.c_float * 10)()
    cb = db.c()
    r = ctx.lib.lyon_gpu_autotune_fill(ctx.h, ctypes.byref(cb), od.data_ptr(), len(opts), 0,
                                       ctypes.byref(best), times, ctypes.byref(nc))
    assert r == T.LYON_OK and nc.value == 10 and min(times) > 0
    assert ctx.lib.lyon_gpu_get_fill_tuning(ctx.h, ctypes.byref(now)) == 0
    assert now.blocks_per_sm == best.blocks_per_sm
    assert best.lanes in (1, 4, 8, 12, 16)
    assert now.lanes == (best.lanes if threads else 0)
