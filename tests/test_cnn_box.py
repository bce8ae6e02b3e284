"""The box kernels of the warm-start network's convolutions (the automatic
choice wherever the tile kernels do not apply): forward, input gradient and
weight gradient against PyTorch fp32, at volumes that divide into 128-voxel
boxes and that do not, channel counts that fill 64- and 32-channel rows and
that leave a part of the last one empty.

Forward and input gradient sum in the gather kernel's order, so their bits are
its bits; against PyTorch, and for the weight gradient (other order, atomics),
FP32 accumulation in a different order: 1e-4 of the maximum.
"""
import pytest
import torch
import torch.nn.functional as F

import xtg
from test_cnn_conv import case, check, conv_path, from_cl, kpad, pack_w, ptr, to_cl

pytestmark = pytest.mark.gpu

SHAPES = [  # nb, Y, X, Z, cin, cout
    (1, 1, 1, 1, 16, 16), (1, 8, 16, 8, 64, 64), (2, 5, 21, 16, 48, 48), (3, 7, 13, 4, 96, 96), (8, 4, 16, 4, 64, 96),
    (1, 3, 9, 33, 112, 48), (2, 6, 10, 4, 32, 80), (1, 17, 18, 8, 160, 64), (5, 2, 3, 5, 80, 32), (1, 2, 130, 6, 48, 112),
    (1, 40, 64, 16, 48, 48), (1, 4, 8, 4, 64, 160), (1, 6, 12, 20, 16, 256)]


@pytest.mark.parametrize("shape", SHAPES)
def test_box_conv(shape):
    lib = xtg.gpu_lib()
    nb, Y, X, Z, cin, cout = shape
    x, w, b = case(shape, 5)
    ref = F.conv3d(x, w, padding=1)
    xd, wd, bd = to_cl(x).to(torch.bfloat16).cuda(), pack_w(w).cuda(), b.float().cuda()
    for epi, want in ((2, ref), (1, ref), (0, torch.relu(ref + b.view(1, -1, 1, 1, 1)))):
        out, gat = (torch.full((nb, Y, X, Z, cout), 7.0, dtype=torch.float32 if epi == 2 else torch.bfloat16, device="cuda")
                    for _ in range(2))
        check(conv_path(lib, xd, wd, bd, out, shape, epi, 1, 0))
        check(conv_path(lib, xd, wd, bd, gat, shape, epi, 1, 1))
        assert torch.equal(out, gat)
        tol = 1e-4 * ref.abs().max() + (0 if epi == 2 else 2 ** -8 * want.abs().max())
        assert torch.max(torch.abs(from_cl(out.float().cpu()) - want)) <= tol


@pytest.mark.parametrize("shape", SHAPES)
def test_box_gradients(shape):
    lib = xtg.gpu_lib()
    nb, Y, X, Z, cin, cout = shape
    x, w, b = case(shape, 6)
    dy = torch.randn(nb, cout, Y, X, Z, generator=torch.Generator().manual_seed(12)).to(torch.bfloat16).float()
    xd, dyd = to_cl(x).to(torch.bfloat16).cuda(), to_cl(dy).to(torch.bfloat16).cuda()
    wtd = pack_w(w.permute(1, 0, 2, 3, 4).contiguous()).cuda()
    out, gat = (torch.empty(nb, Y, X, Z, cin, device="cuda") for _ in range(2))
    for o, path in ((out, 0), (gat, 1)):
        check(lib.xtc_conv3d_path(ptr(dyd), ptr(wtd), None, ptr(o), nb, Y, X, Z, cout, cin, kpad(cout), 2, -1, path))
    assert torch.equal(out, gat)
    ref = torch.nn.grad.conv3d_input(x.shape, w, dy, padding=1)
    assert torch.max(torch.abs(from_cl(out.cpu()) - ref)) <= 1e-4 * torch.max(torch.abs(ref))
    refw = torch.nn.grad.conv3d_weight(x, w.shape, dy, padding=1).permute(2, 3, 4, 1, 0).reshape(27 * cin, cout)
    dw = torch.full((27 * cin + 1, cout), 0.25, device="cuda")  # the call adds; the row past the end stays
    check(lib.xtc_conv3d_wgrad(ptr(xd), ptr(dyd), ptr(dw), nb, Y, X, Z, cin, cout))
    assert torch.all(dw[-1] == 0.25)
    assert torch.max(torch.abs(dw[:-1].cpu() - 0.25 - refw)) <= 1e-4 * torch.max(torch.abs(refw)) + 1e-6
