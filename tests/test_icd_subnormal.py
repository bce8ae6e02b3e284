"""Column visits where neighbouring voxels differ by subnormal amounts, against
the FP64 restatement of a visit (tests/test_icd_cta_sizes.py).

With p = 2 the prior's |d|^(2-p) is 1 for every d but 0, however small; a
logarithm that flushes subnormal differences to 0 must not make it NaN.
Tolerance as there.
"""
import numpy as np
import pytest

import common
import xtg
from test_icd_cta_sizes import visit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mrf_p", [2.0, 1.2])
@pytest.mark.parametrize("order", [xtg.XTG_ORDER_PARALLEL, xtg.XTG_ORDER_SEQUENTIAL])
def test_subnormal_differences(mrf_p, order):
    N, NT, NP = 16, 8, 20
    p = common.params(N=N, NT=NT, NP=NP, zinger=True, nhicd=True)
    p.p = mrf_p
    t, a = common.views(p)
    _, _, y, w = common.data(p, t, a, seed=3, zfrac=0.01)
    rng = np.random.default_rng(2)
    x = np.where(rng.random((1, NT, N, N)) < 0.5, 1e-40, 0.0).astype(np.float32)  # 1e-40: a subnormal
    x[:, :, ::5] = 0.01
    ctx = xtg.Context(p, t, a)
    ctx.set_options(a_mode=xtg.XTG_A_TABLE32, order=order, max_columns=1)
    ctx.upload_sino(y, w)
    ctx.upload_object(x)
    ctx.init_error_sino()
    rx, re = x.astype(np.float64), ctx.error_sino().astype(np.float64)
    items = [(0, 7, 8, -1), (0, 2, 3, -1)]
    ctx.update_columns(1, items)  # a non-finite voxel raises
    got = ctx.object()
    if order == xtg.XTG_ORDER_PARALLEL:  # (the restatement takes even slices first)
        for it in items:
            visit(ctx, ctx.geometry(), p, rx, re, w.astype(np.float64), [np.arange(NP, dtype=np.int32)], 1, it)
        assert np.max(np.abs(got - rx)) <= 1e-4 * np.abs(rx).max()
    assert np.isfinite(got).all()
    ctx.close()
