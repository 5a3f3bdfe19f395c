"""Training calls whose host arrays come through the pinned chunks (16 MB and
more) while the forward runs on the other stream: loss, gradient and updated
weights equal, bit for bit, those of the same calls on pinned host arrays,
which are copied directly.  Two sets of inputs one after the other on the
same network, so that a chunk used again too early or a missing wait shows.
"""
import numpy as np
import pytest
import torch

from test_gpu_unet import R

pytestmark = pytest.mark.gpu


def inputs(seed, B, Z, Y, X):
    rng = np.random.default_rng(seed)
    f = lambda *s: rng.standard_normal(s, dtype=np.float32)
    m = (rng.random((B, Z, Y, X), dtype=np.float32) < 0.8).astype(np.float32)
    return f(B, Z, Y, X, 4), f(B, Z, Y, X), m, f(B, Z, Y, X, 7)


def pinned(a):
    return torch.from_numpy(a).pin_memory().numpy()


def calls(pkg, shape, kind, pin):
    B, Z, Y, X = shape
    net = pkg.UNet(X, Y, Z, B)
    net.set_params(R.he_init(15).astype(np.float32))
    out = []
    for seed in (16, 17, 16):
        x, t, m, a7 = (pinned(a) if pin else a for a in inputs(seed, *shape))
        if kind == "grad":
            out += net.grad(x, t, m)
        else:
            out += net.train_sys(x, t, m, a7, c=1.0, w_mse=0.1, w_res=1.0, lr=1e-3, want_grad=True)
            out.append(net.get_params())
    net.close()
    return out


@pytest.mark.parametrize("shape,kind", [((1, 64, 64, 128), "train_sys"),  # only the second upload in chunks
                                        ((2, 60, 68, 132), "train_sys"),  # both, last chunks partly filled
                                        ((1, 64, 128, 256), "grad")])     # targets and mask exactly 16 MB
def test_chunked_training_arrays(gpu_lib, pkg, shape, kind):
    a, b = calls(pkg, shape, kind, False), calls(pkg, shape, kind, True)
    assert len(a) == len(b)
    for p, q in zip(a, b):
        assert np.isfinite(p).all()
        assert np.asarray(p).tobytes() == np.asarray(q).tobytes()
