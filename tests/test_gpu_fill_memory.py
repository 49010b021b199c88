"""A fill takes sweep heaps for the paths of its batch, not for all that the GPU could sweep at once."""

import pytest

from lyon_gb300 import workloads
from lyon_gb300 import tessellation as T
from oracle import lyon_oracle as orc

import numpy as np

pytestmark = pytest.mark.gpu


def test_memory_of_a_small_fill():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    torch.cuda.synchronize()
    batch, opts = workloads.glyph_fill(300, seed=5)
    od = T.upload_options(opts, 0)
    c = T.Context(0)
    try:
        free = []
        for n in (1, 2, 3, 100, 300):
            part = batch.head(n)
            db = T.DeviceBatch.upload(part, 0)
            torch.cuda.synchronize()
            before = torch.cuda.mem_get_info()[0]
            res = T.tessellate_paths("fill", db, od, len(opts), 32, T.INDEX_PER_PATH, 0, c)
            c.synchronize()
            free.append(before - torch.cuda.mem_get_info()[0])
            ref = orc.batch("fill", part, opts, 32, 8)
            assert np.array_equal(res.indices().cpu().numpy().view(np.uint32), ref["indices"])
        print(free)
        assert free[0] < 64 << 20 and sum(free) < 512 << 20
    finally:
        c.close()
