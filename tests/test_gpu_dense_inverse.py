"""Dense inverse (the AMG coarsest level) at the sizes where its register tiling changes,
against the CPU oracle bit for bit; random matrices, so that most pivots swap rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 32, 33, 64, 65, 96, 97, 127, 128, 129])
def test_dense_inverse_sizes(n):
    from msg123_b200.solver import dense_inverse
    from oracle.oracle import dense_inverse as cpu_inverse
    a = np.random.default_rng(n).standard_normal((n, n))
    assert np.array_equal(dense_inverse(a), cpu_inverse(a))
