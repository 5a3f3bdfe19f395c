"""The U-Net's convolutions and weight gradients at the sizes where their
tilings change: several tiles along x and y, ragged last tiles, both pipeline
depths, several slices of the weight gradient; and the chunked copies of
large host arrays.

Tolerances: those of the comparison with the reference at small sizes
(forward max |y - y_ref| <= 2e-2 max |y_ref| with the BF16-rounding reference;
gradient cosine per layer >= 0.999 with it).  The same item alone or in a
batch gives the same bits, so the chunked path is compared with equality.
"""
import numpy as np
import pytest

from test_gpu_unet import R, batch, layer_slices

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 4, 4, 4), (1, 4, 4, 132), (1, 4, 12, 68), (2, 4, 36, 20), (1, 20, 4, 8),
                                   (1, 4, 4, 260)])
def test_forward_tilings(gpu_lib, pkg, shape):
    B, Z, Y, X = shape
    net = pkg.UNet(X, Y, Z, B)
    p = R.he_init(7).astype(np.float32)
    net.set_params(p)
    x, _, _ = batch(8, B, Z, Y, X)
    y = net.forward(x)
    yr, _ = R.forward(p.astype(np.float64), x.astype(np.float64), q=R.bf16)
    assert np.abs(y - yr).max() <= 2e-2 * np.abs(yr).max()


@pytest.mark.parametrize("shape", [(1, 4, 12, 68), (1, 8, 16, 72), (2, 4, 4, 20)])
def test_gradient_tilings(gpu_lib, pkg, shape):
    B, Z, Y, X = shape
    net = pkg.UNet(X, Y, Z, B)
    p = R.he_init(9).astype(np.float32)
    net.set_params(p)
    x, t, m = batch(10, B, Z, Y, X)
    loss, g = net.grad(x, t, m)
    l_bf, g_bf = R.loss_grad(p.astype(np.float64), x.astype(np.float64), t.astype(np.float64), m.astype(np.float64),
                             q=R.bf16)
    assert abs(loss - l_bf) <= 2e-2 * l_bf
    for name, a, b in layer_slices():
        ga, gb = g[a:b].astype(np.float64), g_bf[a:b]
        if name == "c0":  # the 12 zero input channels carry no gradient
            keep = np.zeros((16, 27, 16), bool)
            keep[:, :, :4] = True
            keep = np.concatenate([keep.ravel(), np.ones(16, bool)])
            ga, gb = ga[keep], gb[keep]
        cos = ga @ gb / (np.linalg.norm(ga) * np.linalg.norm(gb))
        assert cos >= 0.999, (name, cos)


def test_large_host_arrays(gpu_lib, pkg):
    """25 MB of input (chunks through pinned memory, the last one partly
    filled) against the same items one by one (8 MB, one copy each)."""
    Z, Y, X = 64, 64, 128
    p = R.he_init(11).astype(np.float32)
    x, _, _ = batch(12, 3, Z, Y, X)
    one, three = pkg.UNet(X, Y, Z, 1), pkg.UNet(X, Y, Z, 3)
    one.set_params(p)
    three.set_params(p)
    y3 = three.forward(x)
    for b in range(3):
        assert np.array_equal(y3[b], one.forward(x[b:b + 1])[0]), b
