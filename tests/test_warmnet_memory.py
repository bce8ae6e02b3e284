"""The network after a call whose buffers did not fit in device memory: the call
reports it, and calls of an earlier shape work as before (their buffers may have
been given up for the larger ones)."""
import ctypes as C

import pytest

import xtg

pytestmark = pytest.mark.gpu


def test_shape_after_one_that_did_not_fit():
    import torch

    shape = (1, 16, 40, 16)
    g = torch.Generator(device="cuda").manual_seed(3)
    fbp, icd, true = (0.02 * torch.rand(shape, device="cuda", generator=g) for _ in range(3))
    net = xtg.WarmNet(seed=5)
    want, out = torch.empty(shape, device="cuda"), torch.empty(shape, device="cuda")
    net.forward(fbp, icd, want, shape)
    loss = net.backward(fbp, icd, true, shape)
    # 4 G voxels: 256 GB for one level's activations alone; refused before anything runs
    lib = xtg.gpu_lib()
    p = lambda v: C.c_void_p(v.data_ptr())  # noqa: E731
    for _ in range(2):
        rc = lib.xtc_net_forward(net.h, p(fbp), p(icd), p(out), 1, 4096, 2048, 512)
        assert rc == -2, lib.xtg_last_error()
        net.forward(fbp, icd, out, shape)
        torch.cuda.synchronize()
        assert torch.equal(out, want)
        assert abs(net.backward(fbp, icd, true, shape) - loss) <= 1e-6 * loss
    net.close()
