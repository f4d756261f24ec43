"""An output array longer than the sample's field is zero behind it, whatever was in its memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_output_behind_the_field_is_zero():
    from msg123_b200.learned import Cnn
    shape, rng = (12, 10, 8), np.random.default_rng(2)
    n, more = 960, 5000
    cnn = Cnn(seed=1)
    cnn.add_sample(shape, rng.standard_normal((n, 16)).astype(np.float32), np.zeros(n, np.float32))
    for call in (lambda k: cnn.infer(0, k), lambda k: cnn.loss_grad(0, want_grad=False, want_out=True, n=k)[2]):
        want = call(n)
        for _ in range(8):
            used = [np.full(more, 7.0, np.float32) for _ in range(8)]
            del used
            got = call(more)
            assert np.array_equal(got[:n], want) and not got[n:].any()
    cnn.close()
