"""The bin-pair-table projector against the table-free one over the shapes its
kernel splits differently: 4, 8 and 16 lanes per pair and their remainders, odd
bin counts (a last pair of one bin), z-lines with and without 16-byte
alignment, several detector rows per slice, voxels wider than a bin, several
frames, fewer views than a CTA takes, an axis off centre.

A x and e are equal bit for bit and the FP64 cost to 1e-13 (its atomic order
varies).  An infinite voxel reaches the bins its column reaches and no others.
"""
import numpy as np
import pytest

import common
import xtg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,NT,NP,n_time,dxy,dz,rot", [
    (16, 2, 5, 1, 1.0, 1.0, None), (21, 4, 16, 1, 1.0, 1.0, None), (33, 16, 9, 1, 1.0, 1.0, 15.2),
    (24, 18, 20, 1, 1.0, 1.0, None), (27, 27, 12, 1, 1.0, 1.0, None), (40, 32, 31, 1, 1.0, 1.0, None),
    (19, 36, 10, 1, 1.0, 1.0, None), (32, 64, 24, 1, 1.0, 1.0, None), (16, 71, 11, 1, 1.0, 1.0, None),
    (20, 130, 9, 1, 1.0, 1.0, None), (48, 24, 20, 1, 2.0, 2.0, None), (45, 12, 10, 1, 3.0, 1.0, None),
    (32, 8, 48, 4, 1.0, 1.0, None)])
def test_table_projector_equals_gather(N, NT, NP, n_time, dxy, dz, rot):
    p = common.params(N=N, NT=NT, NP=NP, n_time=n_time, dxy=dxy, dz=dz, rot=rot, zinger=True, positivity=0)
    t, a = common.views(p)
    rng = np.random.default_rng(N + NT)
    y = rng.normal(0.3, 0.2, (NP, N, NT)).astype(np.float32)
    w = rng.uniform(10, 1000, y.shape).astype(np.float32)
    d = rng.normal(0, 0.02, (N, NT)).astype(np.float32)
    out = []
    for kind in (xtg.XTG_PROJ_AUTO, xtg.XTG_PROJ_GATHER):
        c = xtg.Context(p, t, a)
        c.set_projector(kind)
        c.upload_sino(y, w, d)
        x = np.random.default_rng(7).normal(0.01, 0.01, c.obj_shape).astype(np.float32)
        c.upload_object(x)
        ax = c.forward_project()
        c.init_error_sino()
        e = c.error_sino()
        cost = c.cost() + c.resync_fp64()
        r = c.error_sino()
        x[-1, c.N_z // 2, c.N_y // 2, c.N_x // 3] = np.inf
        c.upload_object(x)
        out.append((ax, e, r, c.forward_project(), cost, c.projector()))
        c.close()
    u, v = out
    assert u[5][0] == xtg.XTG_PROJ_TABLE and v[5] == (xtg.XTG_PROJ_GATHER, 0)
    for q in range(4):
        assert np.array_equal(u[q], v[q], equal_nan=True), q
    assert np.isinf(u[3]).any() and np.isfinite(u[3]).any()
    assert u[4] == pytest.approx(v[4], rel=1e-13)
