"""The network convolutions' halo tiles (8 z x 16 x of one y-row, nine taps from
one box): volumes that divide into them and that end inside one, one and two
tiles a CTA, channel counts of one and several 32- and 64-channel chunks, and
planes on both sides of the rule that chooses them.  Same comparisons and
tolerances as for the boxes: forward and input gradient have the gather
kernel's bits; FP32 accumulation in another order, 1e-4 of the maximum, else.
"""
import pytest

import test_cnn_box as box

pytestmark = pytest.mark.gpu

SHAPES = [  # nb, Y, X, Z, cin, cout
    (1, 3, 16, 8, 64, 48), (1, 3, 17, 9, 48, 64), (2, 9, 32, 16, 32, 32), (1, 7, 33, 15, 80, 48), (1, 5, 48, 24, 112, 64),
    (2, 30, 31, 7, 96, 96), (1, 2, 5, 3, 128, 128), (1, 4, 64, 40, 160, 96), (1, 6, 16, 8, 256, 16), (1, 12, 40, 8, 16, 256),
    (3, 64, 4, 32, 48, 48)]


@pytest.mark.parametrize("shape", SHAPES)
def test_halo_conv(shape):
    box.test_box_conv(shape)


@pytest.mark.parametrize("shape", SHAPES)
def test_halo_gradients(shape):
    box.test_box_gradients(shape)
