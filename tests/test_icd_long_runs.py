"""Columns whose entry runs nearly fill an SM's shared memory, against the FP64
restatement of a column visit (tests/test_icd_cta_sizes.py).

10,600 views give runs of about 25,500 entries (204 KB); the partial sums of a
1024-thread CTA over 128 rows (32 KB) no longer fit beside them, those of a
256-thread one (8 KB) do.  With one column in flight the CTA size rule would take
the largest.  Tolerance as there.
"""
import numpy as np
import pytest

import common
import xtg
from test_icd_cta_sizes import visit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("amode", [xtg.XTG_A_TABLE32, xtg.XTG_A_FP16])
def test_run_beside_partial_sums(amode):
    N, NT, NP = 16, 128, 10600
    p = common.params(N=N, NT=NT, NP=NP, zinger=True, nhicd=True)
    t, a = common.views(p)
    rng = np.random.default_rng(11)
    y = rng.normal(0.1, 0.02, (NP, N, NT)).astype(np.float32)
    w = rng.uniform(500, 1500, y.shape).astype(np.float32)
    x = rng.uniform(0.0, 0.02, (1, NT, N, N)).astype(np.float32)
    ctx = xtg.Context(p, t, a)
    ctx.set_options(a_mode=amode, max_columns=1)
    ctx.upload_sino(y, w)
    ctx.upload_object(x)
    ctx.init_error_sino()
    views = [np.arange(NP, dtype=np.int32)]
    items = [(0, 8, 7, -1), (0, 2, 3, -1)]
    rx, re = x.astype(np.float64), ctx.error_sino().astype(np.float64)
    ctx.update_columns(2, items)
    for it in items:
        visit(ctx, ctx.geometry(), p, rx, re, w.astype(np.float64), views, 2, it)
    tol = (1e-4 if amode == xtg.XTG_A_TABLE32 else 1e-3) * np.abs(rx).max()  # FP16 entries: 5e-4 relative
    assert np.max(np.abs(ctx.object() - rx)) <= tol
    assert np.max(np.abs(ctx.error_sino() - re)) <= 4 * tol
    ctx.close()
