"""Training passes of the learned guess (loss, gradient, forward output) at grid sizes around
their 16 x 8 x 4 tiles, against the float64 reference with BF16-rounded weights and inputs.
Activations and output gradients are rounded to BF16 (2^-9 relative) at each of the four
layers, so 3e-2 relative, the bound of the package's other gradient tests, covers them."""
import numpy as np
import pytest

from oracle import cnn_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (16, 8, 4), (17, 9, 5), (15, 7, 3), (33, 1, 9), (1, 20, 2), (40, 23, 11)],
                         ids=str)
def test_cnn_gradient_tiles(shape):
    from msg123_b200.learned import Cnn, unpack
    nx, ny, nz = shape
    n = nx * ny * nz
    rng = np.random.default_rng(n)
    x = np.zeros((nz, ny, nx, 16), np.float32)
    x[..., :7] = rng.standard_normal((nz, ny, nx, 7))
    y = (0.3 * rng.standard_normal((nz, ny, nx))).astype(np.float32)
    layers = []
    for l in range(4):
        W, b = np.zeros((27, 16, 16), np.float32), np.zeros(16, np.float32)
        co, ci = (1 if l == 3 else 16), (7 if l == 0 else 16)
        W[:, :co, :ci] = 0.15 * rng.standard_normal((27, co, ci))
        b[:co] = 0.05 * rng.standard_normal(co)
        layers.append((W, b))
    cnn = Cnn(seed=1)
    cnn.set_weights(np.concatenate([np.concatenate([W.reshape(-1), b]) for W, b in layers]).astype(np.float32))
    cnn.add_sample(shape, x.reshape(-1, 16), y.reshape(-1))
    loss, grad, out = cnn.loss_grad(0, want_out=True, n=n)
    ref_loss, ref_out, ref_grads = cnn_ref.loss_and_grad(layers, x, y)
    assert np.linalg.norm(out - ref_out.reshape(-1)) <= 3e-2 * np.linalg.norm(ref_out)
    assert abs(loss - ref_loss) <= 3e-2 * ref_loss
    for l, ((gw, gb), (rw, rb)) in enumerate(zip(unpack(grad), ref_grads)):
        co, ci = (1 if l == 3 else 16), (7 if l == 0 else 16)
        for a, r in ((gw[:, :co, :ci], rw[:, :co, :ci]), (gb[:co], rb[:co])):
            assert np.linalg.norm(a - r) <= 3e-2 * np.linalg.norm(r) + 1e-12
    cnn.close()
