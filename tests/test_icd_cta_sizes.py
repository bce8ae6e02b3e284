"""The ICD column kernel at every CTA size its launch rule picks, against an
FP64 numpy restatement of one column visit.

One column at a time (max_columns = 1), so the visit order is the list's and
nothing is stale: theta over the column's footprint with the
generalized-Huber weight (XT_VoxUpdate.c:20-51), the qGGMRF surrogate step
(XT_ICD_update.c:79-179) for the even then the odd slices, zero skipping from
the second iteration (XT_VoxUpdate.c:208-232), e -= A delta_x.  With one column
in flight the rule takes the smallest CTA whose threads have at most eight
row groups each, up to 1024 threads, so rows x views set the size.

Tolerance: theta sums up to a few thousand FP32 terms of both signs (relative
error below 1e-5 of the sum of magnitudes) and the surrogate weights come from
approximate instructions (a few 1e-6 each); a step is at most the object's
range, so 1e-4 of that range bounds three visits to each column.
"""
import numpy as np
import pytest

import common
import xtg

pytestmark = pytest.mark.gpu


def visit(ctx, g, p, x, e, w, views, it, item):
    """Updates x [N_time][N_z][N_y][N_x] and e in place for item (f, row, col, block)."""
    f, row, col, blk = (int(v) for v in item)
    zo, nz = g.zovl, g.N_z
    zb, ze = (0, nz - 1) if blk < 0 else (blk * g.zstep, nz - 1 if blk == g.nzb - 1 else (blk + 1) * g.zstep - 1)
    vals, idx, cnt = ctx.amatrix(np.full(len(views[f]), row), np.full(len(views[f]), col), views[f])
    ent = [(pv, idx[i, s], float(vals[i, s]) * g.delta_t) for i, pv in enumerate(views[f]) for s in range(cnt[i])]
    pv, bi, a = np.array([t[0] for t in ent]), np.array([t[1] for t in ent]), np.array([t[2] for t in ent])
    t0, t1 = zb * zo, (ze + 1) * zo
    ev, wv = e[pv, bi, t0:t1], w[pv, bi, t0:t1]
    z = np.abs(ev) * np.sqrt(wv)
    we = np.where(z < g.T, wv, g.T * g.delta * np.sqrt(wv) / np.maximum(np.abs(ev), 1e-300))
    th1 = -(a[:, None] * ev * we).sum(0).reshape(-1, zo).sum(1)
    th2 = (a[:, None] ** 2 * we).sum(0).reshape(-1, zo).sum(1)

    def coef(d, sq, sqp, c):
        t = np.abs(d) ** (2 - g.MRF_P) / sqp
        return (2 - (2 - g.MRF_P) * t / (c + t)) / ((c + t) * sq) if d else 2 / (sq * c)

    dx = np.zeros(ze - zb + 1)
    for par in (0, 1):
        for zz in range(zb, ze + 1):
            if zz % 2 != par:
                continue
            v, num, den, pos = x[f, zz, row, col], 0.0, 0.0, False
            for q in range(27):
                dz, dy, dc = q // 9 - 1, q // 3 % 3 - 1, q % 3 - 1
                if q == 13 or not (0 <= zz + dz < nz and 0 <= row + dy < g.N_y and 0 <= col + dc < g.N_x):
                    continue
                u = x[f, zz + dz, row + dy, col + dc]
                b = g.SF[q] * coef(v - u, g.Sigma_S_Q, g.Sigma_S_Q_P, g.C_S)
                num, den, pos = num + b * u, den + b, pos or u > 0
            for f2 in (f - 1, f + 1):
                if 0 <= f2 < g.N_time:
                    u = x[f2, zz, row, col]
                    b = g.TF * coef(v - u, g.Sigma_T_Q, g.Sigma_T_Q_P, g.C_T)
                    num, den, pos = num + b * u, den + b, pos or u > 0
            if v == 0 and it > 1 and not pos:
                continue
            n = v + g.alpha * ((num + th2[zz - zb] * v - th1[zz - zb]) / (den + th2[zz - zb]) - v)
            n = max(n, 0.0) if p.positivity else n
            dx[zz - zb] = n - v
            x[f, zz, row, col] = n
    np.subtract.at(e, (pv, bi, slice(t0, t1)), a[:, None] * np.repeat(dx, zo)[None, :])
    return dx


# N, N_t, views, frames, dz: row groups (entries x threads per entry) from
# about 40 (64 threads) to over 8192 (1024 threads), 16-byte and single rows
@pytest.mark.parametrize("N,NT,NP,n_time,dz,threads", [
    (24, 4, 24, 1, 1.0, 1), (24, 16, 80, 1, 1.0, 1), (20, 16, 200, 1, 1.0, 1), (20, 32, 256, 1, 1.0, 1),
    (16, 64, 400, 1, 1.0, 1), (20, 128, 128, 1, 1.0, 1),
    (20, 8, 96, 3, 1.0, 1), (24, 16, 96, 2, 4.0, 2), (16, 40, 60, 1, 1.0, 5),
    (20, 3, 40, 1, 1.0, 1), (20, 27, 64, 2, 1.0, 1), (16, 31, 200, 1, 1.0, 1), (18, 6, 48, 1, 1.0, 3)])
@pytest.mark.parametrize("amode", [xtg.XTG_A_TABLE32, xtg.XTG_A_FP32])
def test_column_visits_match_restatement(N, NT, NP, n_time, dz, threads, amode):
    p = common.params(N=N, NT=NT, NP=NP, n_time=n_time, dz=dz, zinger=True, nhicd=True, threads=threads * n_time)
    t, a = common.views(p, (4, NP // n_time) if n_time > 1 else None)
    x0, ax, y, w = common.data(p, t, a, seed=7, zfrac=0.01)
    ctx = xtg.Context(p, t, a)
    ctx.set_options(a_mode=amode, max_columns=1)
    ctx.upload_sino(y, w)
    rng = np.random.default_rng(3)
    xs = (x0 * rng.uniform(0.8, 1.2, x0.shape) * (rng.random(x0.shape) > 0.1)).astype(np.float32)
    ctx.upload_object(xs)
    ctx.init_error_sino()
    g = ctx.geometry()
    fov = xtg.host_geometry(p, t, a)[3]
    views = [np.nonzero(fov == f)[0].astype(np.int32) for f in range(n_time)]
    items = [(f, r, c, -1) for f, r, c in zip(rng.integers(0, n_time, 6), rng.integers(0, N, 6), rng.integers(0, N, 6))]
    items += [(0, 0, 0, -1), (n_time - 1, N - 1, N // 2, -1), items[0], (0, N // 2, N // 2, -1), (0, N // 2, N // 2 + 1, -1)]
    rx, re, rw = xs.astype(np.float64), ctx.error_sino().astype(np.float64), ctx.weight().astype(np.float64)
    for lst in (items, [(f, r, c, k % g.nzb) for k, (f, r, c, _) in enumerate(items)]):
        st = ctx.update_columns(2, lst)
        last = {}
        for it in lst:
            last[it] = visit(ctx, g, p, rx, re, rw, views, 2, it)
        assert st.columns == len(lst)
        assert st.voxel_updates + st.zero_skipped == sum(len(last[it]) for it in lst)
        top = np.abs(rx).max()
        assert np.max(np.abs(ctx.object() - rx)) <= 1e-4 * top
        assert np.max(np.abs(ctx.error_sino() - re)) <= 1e-4 * top * 4 * max(1.0, g.delta_t)
        m = ctx.magmap()
        for f, r, c, b in last:
            if b >= 0 and list(k[:3] for k in last).count((f, r, c)) == 1:
                assert abs(m[f, b, r, c] - np.abs(last[f, r, c, b]).sum()) <= 1e-4 * top * g.N_z
    ctx.close()
