"""The FBP start with an object-support disk, and on grids that fill the GPU
with whole tiles, against the FP64 restatement (tests/fbp_check.py).

Small disks leave most tiles empty, one off the tile grid cuts others; the
larger grids launch enough CTAs that no two warps share an image row, whose
tiles reach the most bins (views at 45 and 135 degrees).  Tolerance as in
tests/test_fbp_shapes.py.
"""
import numpy as np
import pytest

import common
import fbp_check
import xtg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,NT,NP,n_time,radius", [
    (80, 5, 20, 1, 11.0), (70, 20, 20, 1, 35.0), (96, 40, 12, 1, 9.5), (50, 66, 9, 2, 0.9), (40, 7, 9, 1, 0.1),
    (337, 70, 4, 1, 168.0), (450, 24, 4, 2, 500.0), (510, 3, 16, 4, 255.0)])
def test_fbp_in_a_disk(N, NT, NP, n_time, radius):
    p = common.params(N=N, NT=NT, NP=NP, n_time=n_time, positivity=N % 2)
    p.radius_obj = radius
    t, a = common.views(p)
    if n_time > 1:
        a = np.tile(a[::n_time], n_time)  # each frame over 180 degrees
    rng = np.random.default_rng(N)
    y = rng.normal(0.5, 0.3, (NP, N, NT)).astype(np.float32)
    ctx = xtg.Context(p, t, a)
    ctx.upload_sino(y, np.ones_like(y))
    ctx.upload_object(np.full(ctx.obj_shape, 7, np.float32))
    ctx.init_fbp()
    ref = fbp_check.fbp(p, t, a, y)
    assert np.max(np.abs(ctx.object() - ref)) <= 1e-4 * max(np.abs(ref).max(), 1e-3)
    ctx.close()
