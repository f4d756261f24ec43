"""DILU factorisation and solve by tile sweeps against the oracle's sequential loops, bit for
bit, at sizes around the 16 x 8 column tiles: one cell, one column, one tile exactly, one cell
more, single rows and layers, several tiles each way, and more cells than one block's share."""
import numpy as np
import pytest

from msg123_b200.config import make_config
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 2), (1, 1, 40), (16, 8, 5), (17, 9, 3), (15, 7, 9), (130, 1, 4), (1, 67, 4),
                                   (5, 40, 2), (33, 25, 2), (48, 47, 21), (97, 83, 37)], ids=str)
def test_dilu_sweep_bitexact(shape):
    from msg123_b200.solver import GpuSolver
    p = make_config("hetero", shape=shape, seed=4, precon_type=0)
    rng = np.random.default_rng(7)
    o = Oracle(p)
    o.init_state()
    o.set_state(head_new=p.head0 + 0.01 * rng.standard_normal(p.ncalc))
    d, lu, r = o.make_matvec()
    o.set_system(d, lu, r)
    with GpuSolver(p) as g:
        g.set_system(d, lu, r)
        for _ in range(3):          # again on the same context: the hand-over slots are empty again
            v = rng.standard_normal(p.ncalc)
            assert np.array_equal(g.precond(v), o.precond(v))
    o.close()
