"""NHICD thresholds and selections at map sizes where the selection kernel
splits a map differently, bit for bit against a NumPy restatement.

The 5x5 filter adds its 25 products in the reference's order in FP32
(ComputeVSC, XT_NHICD.c:128-162), the threshold is the kth smallest filtered
value (RandomizedSelect, XT_NHICD.c:63-126).  A map is shared by 1, 4 or 8 CTAs
(up to 1024 and 4096 values, above); its keys are filtered in the kernel, read
from the filtered map, or (over 49152 a CTA) left there; the last CTA's share is
ragged or empty where the size does not divide.  Maps with ties and many zeros,
and values of a narrow range, whose leading bits agree.
"""
import ctypes as C

import numpy as np
import pytest

import common
import xtg

pytestmark = pytest.mark.gpu

H = np.array([[0.0064, 0.0432, 0.08, 0.0432, 0.0064], [0.0432, 0.2916, 0.54, 0.2916, 0.0432],
              [0.08, 0.54, 1.0, 0.54, 0.08], [0.0432, 0.2916, 0.54, 0.2916, 0.0432],
              [0.0064, 0.0432, 0.08, 0.0432, 0.0064]], np.float32)


def restated(m, kth):
    """thresholds [maps] and selections [maps][ny][nx] of m [maps][ny][nx]"""
    ny, nx = m.shape[1:]
    q = np.pad(m, ((0, 0), (2, 2), (2, 2)))  # (added zeros change no sum of non-negative terms)
    f = np.zeros_like(m)
    for i in range(5):
        for j in range(5):
            f = f + H[i, j] * q[:, i:i + ny, j:j + nx]
    flat = f.reshape(len(m), -1)
    thr = np.array([np.partition(v, k - 1)[k - 1] for v, k in zip(flat, kth)], np.float32)
    return thr, (f > thr[:, None, None]).astype(np.uint8)


def maps(rng, kind, shape):
    if kind == "ties":  # a few values, most of them 0
        return rng.choice(np.array([0, 0, 0, 0.25, 0.5, 1.0], np.float32), shape)
    if kind == "narrow":
        return (1 + 1e-5 * rng.random(shape)).astype(np.float32)
    m = np.exp(rng.normal(-7, 1, shape)).astype(np.float32)
    return m * (rng.random(shape) > 0.2)


@pytest.mark.parametrize("n,ny,nx", [(1, 1, 7), (3, 32, 32), (1, 33, 33), (3, 47, 53), (1, 64, 64), (2, 65, 65), (4, 128, 128),
                                     (70, 40, 101), (16, 256, 256), (2, 301, 299), (1, 512, 768), (1, 701, 699)])
@pytest.mark.parametrize("kind", ["wide", "ties", "narrow"])
def test_thresholds_and_selection(n, ny, nx, kind):
    import torch

    rng = np.random.default_rng(ny * nx + n)
    m = maps(rng, kind, (n, ny, nx)).astype(np.float32)
    lib, pl = xtg.gpu_lib(), ny * nx
    for k in (1, max(1, pl // 2), max(1, pl - pl // 10), pl):
        kth = np.full(n, k, np.int32)
        kth[-1] = max(1, k - 1)  # (ranks differ from map to map)
        d = torch.from_numpy(m).cuda()
        thr = torch.full((n,), -1.0, device="cuda")
        sel = torch.full((n, ny, nx), 7, dtype=torch.uint8, device="cuda")
        p = lambda v: C.c_void_p(v.data_ptr())  # noqa: E731
        assert lib.xtg_nhicd_threshold_noalloc(p(d), n, ny, nx, kth.ctypes.data_as(C.c_void_p), p(thr), p(sel), None) == 0
        torch.cuda.synchronize()
        want_thr, want_sel = restated(m, kth)
        assert np.array_equal(thr.cpu().numpy(), want_thr)
        assert np.array_equal(sel.cpu().numpy(), want_sel)
        assert np.array_equal(d.cpu().numpy(), m)


@pytest.mark.parametrize("N,threads", [(72, 1), (67, 2)])
def test_iteration_selects_a_tenth(N, threads):
    """Every chunk's selection in an iteration takes a tenth of the columns of every
    (frame, z-block): no two filtered values are the same, no voxel is 0."""
    p = common.params(N=N, NT=8, NP=40, nhicd=True, zinger=False, threads=threads, positivity=0)
    t, a = common.views(p)
    x, _, y, w = common.data(p, t, a, seed=5)
    ctx = xtg.Context(p, t, a)
    ctx.set_options(a_mode=xtg.XTG_A_TABLE32)
    ctx.upload_sino(y, w)
    ctx.upload_object((x + np.random.default_rng(1).normal(0, 1e-3, x.shape)).astype(np.float32))
    ctx.init_error_sino()
    ctx.iteration(1)
    st = ctx.iteration(2)
    assert st.columns == N * N + 10 * ctx.nzb * (N * N // 10)
    ctx.close()


def test_captured_in_a_graph():
    """A size whose kernel has not run before, captured and replayed on new maps."""
    import torch

    rng = np.random.default_rng(9)
    lib = xtg.gpu_lib()
    p = lambda v: C.c_void_p(v.data_ptr())  # noqa: E731
    first = torch.rand(1, 16, 16, device="cuda")
    one, kth1 = torch.zeros(1, device="cuda"), np.array([9], np.int32)
    assert lib.xtg_nhicd_threshold_noalloc(p(first), 1, 16, 16, kth1.ctypes.data_as(C.c_void_p), p(one), None, None) == 0
    n, ny, nx = 2, 300, 301
    d, thr, kth = torch.zeros(n, ny, nx, device="cuda"), torch.zeros(n, device="cuda"), np.full(n, 80000, np.int32)
    g, st = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=st):
        rc = lib.xtg_nhicd_threshold_noalloc(p(d), n, ny, nx, kth.ctypes.data_as(C.c_void_p), p(thr), None,
                                             C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    for _ in range(2):
        m = maps(rng, "wide", (n, ny, nx)).astype(np.float32)
        d.copy_(torch.from_numpy(m))
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(thr.cpu().numpy(), restated(m, kth)[0])
