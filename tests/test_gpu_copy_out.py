"""Device-to-host copies into pageable memory: below and above the size at which several
threads share one, sizes that leave a short last piece, two at the same time."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(16, 16, 8), (256, 64, 32), (257, 71, 37)], ids=str)
def test_state_round_trip(shape):
    from msg123_b200.config import make_config
    from msg123_b200.solver import GpuSolver
    p = make_config("hetero", shape=shape, seed=2)
    rng = np.random.default_rng(0)
    h = [p.head0 + 0.01 * rng.standard_normal(p.ncalc) for _ in range(2)]
    with GpuSolver(p) as a, GpuSolver(p) as b:
        for g, x in ((a, h[0]), (b, h[1])):
            g.init_state(x)
        got = {}
        ts = [threading.Thread(target=lambda k=k, g=g: got.update({k: g.get_state()["head_new"]})) for k, g in ((0, a), (1, b))]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        for k in range(2):
            assert np.array_equal(got[k], h[k])
            assert np.array_equal((a, b)[k].get_state()["head_old"], h[k])
