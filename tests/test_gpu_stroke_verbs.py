"""The verb-parallel stroke against the walk of one path by one warp, byte for byte.

The batched stroke works verb by verb (stroke_verbs.cu) and leaves single paths to the walk
(stroke.cu), which the no-allocation entry point still takes for every path. Both restate the same
stroker with the same operations, so every output is equal in every bit: there is no tolerance.
"""

import ctypes

import numpy as np
import pytest

from lyon_gb300 import _native, workloads
from lyon_gb300 import tessellation as T
from lyon_gb300.options import STROKE_OPTIONS_DTYPE
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


def by_walk(ctx, db, od, num_options, bits, mode, offset=0):
    import torch
    n = db.num_paths
    err = ctypes.create_string_buffer(256)
    cap_v = cap_i = 0
    for _ in range(2):
        v = torch.empty(2 * cap_v + 2, dtype=torch.float32, device="cuda")
        i = torch.empty(cap_i + 1, dtype=torch.int32, device="cuda")
        vo = torch.empty(n + 1, dtype=torch.int64, device="cuda")
        io = torch.empty(n + 1, dtype=torch.int64, device="cuda")
        st = torch.empty(max(n, 1), dtype=torch.int32, device="cuda")
        tv, ti, nf = _native.u64(), _native.u64(), _native.u32()
        torch.cuda.synchronize()
        cb = db.c()
        r = ctx.lib.lyon_gpu_stroke_paths_noalloc(
            ctypes.byref(cb), od.data_ptr(), num_options, bits, mode, offset, v.data_ptr(), cap_v,
            i.data_ptr(), cap_i, vo.data_ptr(), io.data_ptr(), st.data_ptr(), ctypes.byref(tv),
            ctypes.byref(ti), ctypes.byref(nf), None, err, len(err))
        torch.cuda.synchronize()
        if r == T.LYON_OK:
            break
        assert r == T.LYON_ERR_CAPACITY, (r, err.value)
        cap_v, cap_i = tv.value, ti.value
    dt = np.uint16 if bits == 16 else np.uint32
    return dict(v=v.cpu().numpy()[:2 * tv.value].view(np.uint32),
                i=i.cpu().numpy().view(dt)[:ti.value], vo=vo.cpu().numpy(), io=io.cpu().numpy(),
                st=st.cpu().numpy()[:n], failed=nf.value)


def by_verb(ctx, db, od, num_options, bits, mode, offset=0):
    res = T.tessellate_paths("stroke", db, od, num_options, bits, mode, offset, ctx)
    ctx.synchronize()
    vo, io = res.offsets()
    dt = np.uint16 if bits == 16 else np.uint32
    v = (res.vertices().cpu().numpy().reshape(-1).view(np.uint32) if res.total_vertices
         else np.zeros(0, np.uint32))
    i = res.indices().cpu().numpy().view(dt) if res.total_indices else np.zeros(0, dt)
    return dict(v=v, i=i, vo=vo.cpu().numpy(), io=io.cpu().numpy(),
                st=res.statuses().cpu().numpy(), failed=res.num_failed_paths)


def check(ctx, batch, opts, bits=32, mode=T.INDEX_GLOBAL, offset=0):
    db, od = T.DeviceBatch.upload(batch, 0), T.upload_options(opts, 0)
    a = by_walk(ctx, db, od, len(opts), bits, mode, offset)
    b = by_verb(ctx, db, od, len(opts), bits, mode, offset)
    assert np.array_equal(a["st"], b["st"]), np.nonzero(a["st"] != b["st"])[0][:10]
    for k in ("vo", "io"):
        assert np.array_equal(a[k], b[k]), np.nonzero(np.diff(a[k]) != np.diff(b[k]))[0][:10]
    assert a["failed"] == b["failed"]
    assert np.array_equal(a["i"], b["i"])
    # NaN positions (a path may have them) compare by their place, all else by its bits.
    va, vb = a["v"].view(np.float32), b["v"].view(np.float32)
    nan = np.isnan(va)
    assert np.array_equal(nan, np.isnan(vb))
    assert np.array_equal(a["v"][~nan], b["v"][~nan])
    return a


def options(rng, n, tol=None, join=None):
    o = np.zeros(n, STROKE_OPTIONS_DTYPE)
    o["start_cap"] = rng.integers(0, 3, n)
    o["end_cap"] = rng.integers(0, 3, n)
    o["line_join"] = rng.integers(0, 4, n) if join is None else join
    o["line_width"] = rng.choice([0.0, 0.3, 1.0, 5.0, 40.0], n).astype(np.float32)
    o["miter_limit"] = rng.choice([1.0, 2.0, 4.0, 10.0], n).astype(np.float32)
    o["tolerance"] = rng.choice([0.01, 0.1, 1.0, 8.0], n) if tol is None else tol
    return o


def rough_paths(n, seed, max_verbs=40):
    """Paths of one to three sub-paths whose points repeat, nearly repeat or reverse: merges at
    every place of a sub-path, cusps, curves with control points on their ends, empty sub-paths."""
    rng = np.random.default_rng(seed)
    verbs, pts, vo, po = [], [], [0], [0]
    for _ in range(n):
        for _ in range(int(rng.choice([1, 1, 1, 2, 3]))):
            p = rng.uniform(0, 400, 2)
            start = p.copy()
            verbs.append(Verb.BEGIN)
            pts.append(p)
            scale = rng.choice([0.05, 2.0, 60.0])
            for _ in range(int(rng.integers(0, rng.choice([2, 4, max_verbs])))):
                k = int(rng.choice([0, 0, 1, 2]))
                step = rng.normal(0, scale, (k + 1, 2))
                r = rng.random()
                if r < 0.15:
                    step[:] = 0.0
                elif r < 0.3:
                    step *= 1e-3
                elif r < 0.45 and k:
                    step[1:] = 0.0          # control points on the end point
                elif r < 0.55 and k == 2:
                    step[1] = -2 * step[0]  # a cusp, or nearly one
                elif r < 0.65:
                    step[-1] = -step[:-1].sum(0) - rng.normal(0, 1e-2, 2)  # back to the start
                verbs.append(k)
                for s in step:
                    p = p + s
                    pts.append(p)
            if rng.random() < 0.5:
                verbs.append(Verb.CLOSE)
                pts.append(start)
            else:
                verbs.append(Verb.END)
        vo.append(len(verbs))
        po.append(len(pts))
    return PathBatch(np.array(verbs, np.uint8), np.array(pts, np.float32).reshape(-1, 2),
                     np.array(vo, np.uint32), np.array(po, np.uint32))


@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("join", [None, 0, 1, 2, 3])
def test_rough_paths(ctx, seed, join):
    batch = rough_paths(600, seed)
    o = options(np.random.default_rng(seed + 100), batch.num_paths, join=join)
    check(ctx, batch, o)


@pytest.mark.parametrize("bits,mode,offset", [(16, T.INDEX_PER_PATH, 60000),
                                              (16, T.INDEX_GLOBAL, 7),
                                              (32, T.INDEX_PER_PATH, 3), (32, T.INDEX_GLOBAL, 5)])
def test_index_types_and_modes(ctx, bits, mode, offset):
    batch, o = workloads.batched_stroke(500, seed=21)
    a = check(ctx, batch, o, bits, mode, offset)
    if bits == 16:
        assert a["failed"] > 0  # some paths or their ids pass 16 bits: rolled back alike


@pytest.mark.parametrize("tol,make", [(0.02, "curves"), (0.5, "curves"), (0.02, "lines"),
                                      (1.0, "lines")])
def test_generated_scenes(ctx, tol, make):
    if make == "curves":
        batch, o = workloads.batched_stroke(4000, seed=31)
        o["line_join"] = np.arange(len(o)) % 4
        o["start_cap"] = np.arange(len(o)) % 3
        o["tolerance"] = tol
    else:
        batch, o = workloads.map_polylines(20000, seed=32, tolerance=tol)
        o["line_join"] = np.arange(len(o)) % 4
        o["end_cap"] = np.arange(len(o)) % 3
    check(ctx, batch, o)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 257])
def test_small_batches(ctx, n):
    # Windows, tiles and grids that are not full; one shared option record.
    batch = rough_paths(n, 50 + n, max_verbs=100)
    check(ctx, batch, options(np.random.default_rng(n), 1, tol=0.1))


def test_batches_that_outgrow_the_arrays(ctx):
    # A context sizes its arrays by the first batch; larger ones are counted again.
    c = T.Context(0)
    try:
        for n in (3, 2000, 5, 9000):
            batch = rough_paths(n, n, max_verbs=10)
            check(c, batch, options(np.random.default_rng(n), batch.num_paths))
    finally:
        c.close()


def test_broken_paths_and_offsets(ctx):
    good = rough_paths(40, 3)
    o = options(np.random.default_rng(8), 40, tol=0.1)
    rng = np.random.default_rng(9)
    for trial in range(12):
        v, vo, po = good.verbs.copy(), good.verb_offsets.copy(), good.point_offsets.copy()
        pts = good.points.copy()
        at = rng.integers(0, len(v), 6)
        if trial < 4:
            v[at] = rng.integers(0, 9, 6)                       # wrong grammar, unknown verbs
        elif trial < 6:
            pts[rng.integers(0, len(pts), 3)] = [np.nan, np.inf]
        elif trial < 8:
            po[1 + rng.integers(0, 38)] += 2                    # points short, or too many
        elif trial == 8:
            o = o.copy()
            o["tolerance"][::3] = [np.nan, 0.0][trial % 2]
        elif trial == 9:
            pts[rng.integers(0, len(pts), 4)] *= 1e6            # curves of very many steps
        elif trial == 10:
            vo[5], po[5] = vo[6], po[6]                         # an empty path
            v[vo[6]:vo[7]] = good.verbs[vo[6]:vo[7]]
        else:
            vo[20], po[20] = vo[22], po[22]                     # offsets that overlap
        check(ctx, PathBatch(v, pts, vo, po), o)


def test_offsets_from_the_middle_of_a_batch(ctx):
    # A view of paths [7, 30) of a larger batch: the first offset is not 0.
    batch = rough_paths(60, 77)
    o = options(np.random.default_rng(1), 23)
    db = T.DeviceBatch.upload(batch, 0)
    db.verb_offsets, db.point_offsets = db.verb_offsets[7:31], db.point_offsets[7:31]
    db.num_paths = 23
    od = T.upload_options(o, 0)
    a = by_walk(ctx, db, od, 23, 32, T.INDEX_GLOBAL)
    b = by_verb(ctx, db, od, 23, 32, T.INDEX_GLOBAL)
    assert all(np.array_equal(a[k], b[k]) for k in ("st", "vo", "io", "i", "v"))


# ---- attribute records, variable widths and vertex sources ----------------------------------------

def stepped(ctx, batch, opts, how, by_path=False, bits=32, mode=T.INDEX_GLOBAL):
    """One call of the stepped outputs. With `by_path` a last path whose offsets run backwards (it
    strokes to nothing) makes the whole batch go path by path."""
    import torch
    vo, po = batch.verb_offsets, batch.point_offsets
    if by_path:
        vo, po = np.append(vo, vo[-1] - 1), np.append(po, po[-1])
        opts = np.append(opts, opts[-1:]) if len(opts) > 1 else opts
    b = PathBatch(batch.verbs, batch.points, vo.astype(np.uint32), po.astype(np.uint32))
    db, od = T.DeviceBatch.upload(b, 0), T.upload_options(opts, 0)
    rng = np.random.default_rng(5)
    w = torch.from_numpy(rng.uniform(0.3, 2.5, len(b.points)).astype(np.float32)).cuda()
    attrs = torch.from_numpy(rng.uniform(0.5, 2, (len(b.points), 3)).astype(np.float32)).cuda()
    kw = {"records": dict(attributes=True), "widths": dict(widths=w),
          "widths records": dict(widths=w, attributes=True),
          "sources": dict(custom_attributes=attrs),
          "sources records": dict(custom_attributes=attrs, attributes=True),
          "sources widths": dict(custom_attributes=attrs, width_attribute=1),
          "sources widths records": dict(custom_attributes=attrs, width_attribute=2,
                                         attributes=True)}[how]
    torch.cuda.synchronize()
    res = T.tessellate_paths("stroke", db, od, len(opts), bits, mode, 0, ctx, **kw)
    ctx.synchronize()
    n = batch.num_paths
    out = {"st": res.statuses().cpu().numpy()[:n], "failed": np.array(res.num_failed_paths)}
    o = res.offsets()
    out["vo"], out["io"] = o[0].cpu().numpy()[:n + 1], o[1].cpu().numpy()[:n + 1]
    if res.total_vertices:
        v = res.records() if "records" in how else res.vertices()
        out["v"] = v.cpu().numpy()
        if "sources" in how:
            out["src"] = res.sources().cpu().numpy()
            out["attr"] = res.custom_attributes().cpu().numpy()
    if res.total_indices:
        out["i"] = res.indices().cpu().numpy()
    return out


def same_bits(a, b):
    assert a.keys() == b.keys()
    for k in a:
        x, y = a[k], b[k]
        assert x.shape == y.shape, (k, x.shape, y.shape)
        if x.dtype == np.float32:
            nan = np.isnan(x)
            assert np.array_equal(nan, np.isnan(y)), k
            x, y = x[~nan].view(np.uint32), y[~nan].view(np.uint32)
        assert np.array_equal(x, y), (k, np.nonzero(x != y)[0][:8])


STEPPED = ["records", "widths", "widths records", "sources", "sources records", "sources widths",
           "sources widths records"]


@pytest.mark.parametrize("how", STEPPED)
@pytest.mark.parametrize("join", [None, 0, 1, 2, 3])
def test_stepped_rough_paths(ctx, how, join):
    for seed in (11, 12):
        batch = rough_paths(500, seed)
        o = options(np.random.default_rng(seed), batch.num_paths, join=join)
        o["line_width"] = np.maximum(o["line_width"], 0.3)
        same_bits(stepped(ctx, batch, o, how, by_path=True), stepped(ctx, batch, o, how))


@pytest.mark.parametrize("how", STEPPED)
def test_stepped_scenes(ctx, how):
    batch, o = workloads.batched_stroke(600, seed=41)
    o["line_join"] = np.arange(len(o)) % 4
    o["start_cap"] = np.arange(len(o)) % 3
    o["tolerance"] = 0.1
    same_bits(stepped(ctx, batch, o, how, by_path=True), stepped(ctx, batch, o, how))
    batch, o = workloads.map_polylines(1500, seed=42, max_len=300)
    same_bits(stepped(ctx, batch, o, how, by_path=True, bits=16, mode=T.INDEX_PER_PATH),
              stepped(ctx, batch, o, how, bits=16, mode=T.INDEX_PER_PATH))


@pytest.mark.parametrize("n", [1, 2, 33])
def test_stepped_small_batches(ctx, n):
    for how in STEPPED:
        batch = rough_paths(n, 90 + n, max_verbs=120)
        o = options(np.random.default_rng(n), 1, tol=0.05)
        o["line_width"] = 3.0
        same_bits(stepped(ctx, batch, o, how, by_path=True), stepped(ctx, batch, o, how))


@pytest.mark.parametrize("n", [255, 256, 257, 2047, 2048, 2049])
def test_counts_finished_by_one_block(ctx, n):
    # Up to 2,048 paths one block sums paths and, for a tile of 2,048 verbs or fewer as the call
    # before had, the verbs; the batch here has more verbs than that call. At this vertex offset
    # the longer paths pass the range of 16-bit indices and fail.
    rng = np.random.default_rng(n)
    first = rough_paths(3, n)
    check(ctx, first, options(rng, first.num_paths))
    batch = rough_paths(n, n + 1, 12)
    opts = options(rng, batch.num_paths)
    check(ctx, batch, opts)
    check(ctx, batch, opts, 16, T.INDEX_PER_PATH, 65500)


@pytest.mark.parametrize("limit", [1.0, 1.05, 1.5, 4.0])
@pytest.mark.parametrize("width", [0.3, 5.0, 40.0])
def test_clipped_miters(ctx, limit, width):
    # Clipped miters leave sides that are not symmetric, before runs, at cusps and inside irregular
    # verbs: the skip test of the step after each is evaluated, not ruled out by its bound.
    batch = rough_paths(600, int(limit * 100 + width))
    opts = options(np.random.default_rng(5), batch.num_paths, join=1)
    opts["miter_limit"] = limit
    opts["line_width"] = width
    check(ctx, batch, opts)
