"""The FBP start over the shapes its kernels tile differently, against the FP64
restatement (tests/fbp_check.py).

Slices per lane group 16 / 32 / 64 and remainders, rows that do not align to
16 bytes, detector rows summed per slice, voxels wider than a bin (more than
one bin per column step), several frames, an offset, grids smaller than a tile
and bins beyond the detector (an off-centre axis).

Tolerance: FP32 interpolation positions at magnitude N_r are off by a few
units in the last place (2e-5 of a bin at 64 bins), which a ramp-filtered row
of noise turns into 2e-5 of its range per view; sums of views average it.
1e-4 of the image's maximum, as for the golden cases.
"""
import numpy as np
import pytest

import common
import fbp_check
import xtg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,NT,NP,n_time,dxy,dz,rot", [
    (16, 2, 7, 1, 1.0, 1.0, None), (40, 3, 33, 1, 1.0, 1.0, None), (33, 17, 20, 1, 1.0, 1.0, None),
    (48, 16, 64, 1, 1.0, 1.0, 20.3), (37, 27, 50, 1, 1.0, 1.0, None), (64, 32, 91, 1, 1.0, 1.0, None),
    (50, 64, 30, 1, 1.0, 1.0, 27.9), (35, 70, 24, 1, 1.0, 1.0, None), (64, 16, 48, 1, 2.0, 2.0, None),
    (60, 24, 40, 1, 3.0, 1.0, None), (32, 8, 96, 3, 1.0, 1.0, None), (48, 80, 40, 2, 2.0, 2.0, None)])
def test_fbp_matches_checker(N, NT, NP, n_time, dxy, dz, rot):
    p = common.params(N=N, NT=NT, NP=NP, n_time=n_time, dxy=dxy, dz=dz, rot=rot, positivity=N % 2)
    t, a = common.views(p)
    rng = np.random.default_rng(N)
    y = rng.normal(0.5, 0.3, (NP, N, NT)).astype(np.float32)
    d = rng.normal(0.0, 0.05, (N, NT)).astype(np.float32)
    ctx = xtg.Context(p, t, a)
    ctx.upload_sino(y, np.ones_like(y), d)
    ctx.init_fbp()
    ref = fbp_check.fbp(p, t, a, y, d)
    assert np.max(np.abs(ctx.object() - ref)) <= 1e-4 * np.abs(ref).max()
    ctx.close()
