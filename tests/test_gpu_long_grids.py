"""Grids of more rows or layers than a launch has blocks in y or z (65535): the hierarchy and the
preconditioner of a system set by the caller, bit for bit as the oracle's."""
import numpy as np
import pytest

from msg123_b200.config import make_config
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 70001), (1, 270003, 1), (2, 3, 65536)], ids=str)
def test_hierarchy_of_long_grid(shape):
    from msg123_b200.solver import GpuSolver
    kw = dict(precon_type=1, ref_quirks=0, amg_coarse_max=16)
    p = make_config("hetero", shape=shape, seed=3)
    rng = np.random.default_rng(2)
    o = Oracle(p, **kw)
    o.init_state()
    o.set_state(head_new=p.head0 + 0.01 * rng.standard_normal(p.ncalc), delt=3600.0)
    d, lu, r = o.make_matvec()
    o.set_system(d, lu, r)
    v = rng.standard_normal(p.ncalc)
    with GpuSolver(p, **kw) as g:
        g.set_system(d, lu, r)
        assert np.array_equal(g.precond(v), o.precond(v))
    o.close()
