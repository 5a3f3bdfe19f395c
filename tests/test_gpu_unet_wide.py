"""Networks so wide that a row of the convolutions' usual tiles does not fit
shared memory with 96 channels (X from 1704) and with 64 (X from 3920).

Tolerances: those of the comparison at small sizes (forward max |y - y_ref|
<= 2e-2 max |y_ref| with the BF16-rounding reference; loss within 2 %,
gradient cosine per layer >= 0.999 with it).
"""
import numpy as np
import pytest

from test_gpu_unet import R, batch, layer_slices

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("X", [1704, 2048, 3920])
def test_wide_network(gpu_lib, pkg, X):
    B, Z, Y = 1, 4, 4
    net = pkg.UNet(X, Y, Z, B)
    p = R.he_init(13).astype(np.float32)
    net.set_params(p)
    x, t, m = batch(14, B, Z, Y, X)
    y = net.forward(x)
    p64, x64 = p.astype(np.float64), x.astype(np.float64)
    yr, _ = R.forward(p64, x64, q=R.bf16)
    assert np.abs(y - yr).max() <= 2e-2 * np.abs(yr).max()
    loss, g = net.grad(x, t, m)
    l_bf, g_bf = R.loss_grad(p64, x64, t.astype(np.float64), m.astype(np.float64), q=R.bf16)
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
