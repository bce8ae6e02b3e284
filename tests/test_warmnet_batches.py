"""A batch of volumes through the network against the volumes one by one.

Alone, a volume gives every CTA of the first layer's kernels one tile, whose halo
is read whole; sixteen of them give runs of several tiles, which keep rows of the
halo from tile to tile and cross columns and volumes, and sums over several
tiles.  The forward pass is the same bits.  The loss is a mean, so the batch's
gradients are the mean of the volumes': every product and rounding on the way is
the same but for the factor 1/16, a power of two, and only FP32 sums are taken in
another order (1e-6 of the largest term; 2e-5 of the largest gradient bounds
that).  Slices in multiples of 32, 16 and 8, columns that do not fill a tile.
"""
import numpy as np
import pytest

import xtg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Y,X,Z", [(16, 40, 32), (32, 40, 16), (56, 40, 8)])
def test_batch_equals_its_volumes(Y, X, Z):
    import torch

    nb = 16
    g = torch.Generator(device="cuda").manual_seed(Y + Z)
    rnd = lambda: 0.02 * torch.rand(nb, Y, X, Z, device="cuda", generator=g)  # noqa: E731
    fbp, icd, true = rnd(), rnd(), rnd()
    net = xtg.WarmNet(seed=5)
    out = torch.empty_like(icd)
    net.forward(fbp, icd, out, tuple(out.shape))
    loss = net.backward(fbp, icd, true, tuple(out.shape))
    grads = np.array(net.params(1), np.float64)
    one, mean, losses = torch.empty(1, Y, X, Z, device="cuda"), 0.0, []
    for b in range(nb):
        f, q, t = (v[b:b + 1].contiguous() for v in (fbp, icd, true))
        net.forward(f, q, one, tuple(one.shape))
        torch.cuda.synchronize()
        assert torch.equal(one[0], out[b])
        losses.append(net.backward(f, q, t, tuple(one.shape)))
        mean = mean + np.array(net.params(1), np.float64) / nb
    net.close()
    assert abs(loss - np.mean(losses)) <= 1e-6 * abs(loss)
    first = slice(0, 27 * 2 * 32 + 32)  # the first layer's weights and biases
    assert np.max(np.abs(grads[first] - mean[first])) <= 2e-5 * np.abs(mean[first]).max()
    assert np.max(np.abs(grads - mean)) <= 2e-5 * np.abs(mean).max()
