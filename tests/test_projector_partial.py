"""The table projector where device memory is short.

A table of one entry per (column, view, bin), 8 bytes each, is what the projector
may take; its records of two bins are about a tenth larger in all, so where only
the former fits it holds the views that do and the others are projected without.
The values are those of the full table and of the projector without one, bit
for bit; FP64 costs to the order of their sums.  The free memory is set with a
filler buffer; 3 % above the entries' bytes lies between the two sizes.
"""
import numpy as np
import pytest

import common
import xtg

pytestmark = pytest.mark.gpu
GIB = 1 << 30


def project(ctx):
    ctx.init_error_sino()
    return ctx.forward_project(), ctx.error_sino(), ctx.cost(), ctx.resync_fp64(), ctx.error_sino()


def same(a, b):
    for u, v in zip(a, b):
        if isinstance(u, np.ndarray):
            assert np.array_equal(u, v)
        else:
            assert np.allclose(u, v, rtol=1e-12)


@pytest.mark.parametrize("N,NT,NP,n_time", [(256, 32, 512, 1), (200, 13, 600, 4)])
def test_views_that_fit(N, NT, NP, n_time):
    import torch

    p = common.params(N=N, NT=NT, NP=NP, n_time=n_time)
    t, a = common.views(p)
    rng = np.random.default_rng(N)
    y = rng.normal(0.5, 0.1, (NP, N, NT)).astype(np.float32)
    x = rng.uniform(0, 0.02, (n_time, NT, N, N)).astype(np.float32)

    def context():
        c = xtg.Context(p, t, a)
        c.upload_sino(y, np.ones_like(y))
        c.upload_object(x)
        return c

    c = context()
    want = project(c)
    kind, entries = c.projector()
    assert kind == xtg.XTG_PROJ_TABLE
    c.close()
    single = 8 * entries + 8 * (NP * N + 1)
    for room, expect in ((1.03, xtg.XTG_PROJ_TABLE), (0.9, xtg.XTG_PROJ_GATHER)):
        torch.cuda.empty_cache()
        c = context()
        c.cost_running()  # (buffers of the calls below that are not the table's)
        torch.cuda.synchronize()
        # what the table's construction allocates beside it for its counts: a word a row, two a view
        extra = 4 * NP * ((N + 1) // 2) + 8 * NP
        keep = 2 * GIB + int(room * single)
        free = torch.cuda.mem_get_info()[0]
        assert free > keep + extra
        filler = torch.empty(free - keep, dtype=torch.uint8, device="cuda")
        left = torch.cuda.mem_get_info()[0] - 2 * GIB
        assert abs(left - room * single) < 0.02 * single
        got = project(c)
        kind, n = c.projector()
        assert kind == expect
        if expect == xtg.XTG_PROJ_TABLE:
            assert 0.8 * entries < n < entries
        same(got, want)
        c.close()
        del filler
    torch.cuda.empty_cache()
