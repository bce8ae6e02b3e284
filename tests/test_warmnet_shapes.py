"""The network's gradients where its elementwise kernels leave remainders:
voxel counts that do not divide by a block's share, one and several batches,
single-voxel coarsest levels.  Reference, tolerances and their reasons as in
test_warmnet.py."""
import pytest
import torch

import warmnet_ref as ref
import xtg
from test_warmnet import random_params, volumes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 8, 8, 8), (3, 8, 24, 16), (5, 16, 8, 8), (1, 24, 40, 24)])
def test_gradients_match_reference(shape):
    net = xtg.WarmNet(seed=4)
    p = random_params(net, 6)
    net.set_params(p)
    fbp, icd, tgt = volumes(shape, 13)
    out = torch.empty(shape, device="cuda")
    fd, idd, td = fbp.cuda(), icd.cuda(), tgt.cuda()
    net.forward(fd, idd, out, shape)  # first without gradient buffers
    loss = net.backward(fd, idd, td, shape)
    g = torch.from_numpy(net.params(1))
    rloss, ry, rg = ref.loss_and_grads(p, fbp, icd, tgt)
    corr = ry - icd
    assert torch.max(torch.abs(out.cpu() - ry)) <= 2e-2 * float(corr.max() - corr.min())
    assert loss == pytest.approx(rloss, rel=2e-2)
    assert float(torch.dot(g, rg) / (torch.norm(g) * torch.norm(rg))) >= 0.998
    # the head's own gradients: sums of the loss gradient without a rounding on the way
    n = ref.HEAD_C + 1
    assert float(torch.norm(g[-n:] - rg[-n:]) / torch.norm(rg[-n:])) <= 2e-2
    net.close()
