"""Training passes of the learned guess on fields longer in y or z than a launch has blocks there
(65535 tiles of 8 rows or 4 layers): the same field along x, with the taps' axes exchanged, gives
the same numbers.  In a single row of cells a tap off the row adds zeros, so the outputs are the
same bits; the gradient's sums run in another order (FP32, 1e-3 of the norm is hundreds of
times their rounding)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis,n", [(0, 262145), (1, 524289)], ids=["z", "y"])
def test_long_field(axis, n):
    from msg123_b200.learned import Cnn, unpack
    rng = np.random.default_rng(n)
    x = np.zeros((n, 16), np.float32)
    x[:, :7] = rng.standard_normal((n, 7))
    y = (0.3 * rng.standard_normal(n)).astype(np.float32)
    W = (0.15 * rng.standard_normal((4, 3, 3, 3, 16, 16))).astype(np.float32)
    b = (0.05 * rng.standard_normal((4, 16))).astype(np.float32)

    def run(shape, taps):
        flat = np.concatenate([np.concatenate([w.reshape(-1), c]) for w, c in zip(taps, b)])
        with_cnn = Cnn(seed=1)
        with_cnn.set_weights(flat)
        with_cnn.add_sample(shape, x, y)
        loss, grad, out = with_cnn.loss_grad(0, want_out=True, n=n)
        with_cnn.close()
        return loss, unpack(grad), out

    shape = (1, 1, n) if axis == 0 else (1, n, 1)
    loss, grad, out = run(shape, np.ascontiguousarray(W.swapaxes(1 + axis, 3)))
    loss_x, grad_x, out_x = run((n, 1, 1), W)
    assert np.array_equal(out, out_x)
    assert abs(loss - loss_x) <= 1e-12 * loss_x
    for (gw, gb), (rw, rb) in zip(grad, grad_x):
        gw = np.asarray(gw).reshape(3, 3, 3, 16, 16).swapaxes(axis, 2).reshape(27, 16, 16)
        assert np.linalg.norm(gw - rw) <= 1e-3 * np.linalg.norm(rw)
        assert np.linalg.norm(gb - rb) <= 1e-3 * np.linalg.norm(rb)
