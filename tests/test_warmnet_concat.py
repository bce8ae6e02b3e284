"""Inference reads the decoder's concatenations (2x upsampling beside the skip
input) in place: forward output against the PyTorch restatement at volumes with
one, two and three such levels, several batches and ragged z tiles.  Tolerance
and its reason as in test_warmnet.py; the training pass on the same object
afterwards forms the concatenations and has to find its own buffers."""
import pytest
import torch

import warmnet_ref as ref
import xtg
from test_warmnet import random_params, volumes

pytestmark = pytest.mark.gpu


# X = 128, 256, 512: one, two and three decoder levels with rows of 128 voxels
@pytest.mark.parametrize("shape", [(2, 16, 128, 24), (1, 8, 256, 8), (1, 8, 512, 16)])
def test_concatenation_in_place(shape):
    net = xtg.WarmNet(seed=2)
    p = random_params(net, 7)
    net.set_params(p)
    fbp, icd, tgt = volumes(shape, 5)
    out = torch.empty(shape, device="cuda")
    net.forward(fbp.cuda(), icd.cuda(), out, shape)
    loss = net.backward(fbp.cuda(), icd.cuda(), tgt.cuda(), shape)
    rloss, ry, _ = ref.loss_and_grads(p, fbp, icd, tgt)
    corr = ry - icd
    assert torch.max(torch.abs(out.cpu() - ry)) <= 2e-2 * float(corr.max() - corr.min())
    assert loss == pytest.approx(rloss, rel=2e-2)
    net.close()


def test_head_beside_and_inside_the_last_convolution():
    """The fused head needs 16-byte aligned volumes; a volume that is not gets the
    separate head, with the same sums in the same order."""
    shape = (1, 8, 128, 24)
    net = xtg.WarmNet(seed=3)
    net.set_params(random_params(net, 4))
    fbp, icd, _ = volumes(shape, 9)
    n = fbp.numel()
    outs = []
    for off_out, off_icd in ((0, 0), (1, 0), (0, 3)):
        out = torch.empty(n + 8, device="cuda")[off_out:off_out + n]
        base = torch.empty(n + 8, device="cuda")[off_icd:off_icd + n]
        base.copy_(icd.reshape(-1))
        net.forward(fbp.cuda(), base, out, shape)
        outs.append(out.cpu())
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    net.close()
