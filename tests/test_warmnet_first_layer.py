"""The first layer's kernels at every z tile (32, 16, 8 voxels) and with rows
that end inside a tile: the inference's output and the layer's weight gradient
against the PyTorch restatement.  Tolerances and their reasons as in
test_warmnet.py."""
import pytest
import torch

import warmnet_ref as ref
import xtg
from test_warmnet import random_params, volumes

pytestmark = pytest.mark.gpu


# tiles of 4, 8 and 16 x: rows of 8, 24 and 40 voxels leave remainders
@pytest.mark.parametrize("shape", [(1, 8, 8, 32), (2, 8, 24, 16), (1, 16, 40, 8), (1, 8, 8, 96)])
def test_first_layer(shape):
    net = xtg.WarmNet(seed=5)
    p = random_params(net, 9)
    net.set_params(p)
    fbp, icd, tgt = volumes(shape, 3)
    out = torch.empty(shape, device="cuda")
    net.forward(fbp.cuda(), icd.cuda(), out, shape)
    net.backward(fbp.cuda(), icd.cuda(), tgt.cuda(), shape)
    g = torch.from_numpy(net.params(1))
    _, ry, rg = ref.loss_and_grads(p, fbp, icd, tgt)
    corr = ry - icd
    assert torch.max(torch.abs(out.cpu() - ry)) <= 2e-2 * float(corr.max() - corr.min())
    n = 27 * 2 * 32
    assert float(torch.norm(g[:n] - rg[:n]) / torch.norm(rg[:n])) <= 1e-1
    net.close()
