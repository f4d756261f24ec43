"""Small levels of a V-cycle in one cluster launch: FP64 bit for bit against the oracle, the
mixed cycle against it within its storage (BF16 off-diagonals are 2^-9 off, a cycle of a few
sweeps multiplies that by less than ten: 2e-2 of the norm).  Sizes on both sides of a
slice, odd row counts, a first small level near the row limit and one with long rows (whose
operator and transfers do not fit in shared memory), a dense and a smoothed last level, 0 to 3
sweeps."""
import numpy as np
import pytest

from msg123_b200.config import make_config
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sweeps", [0, 1, 2, 3])
@pytest.mark.parametrize("shape,nlevel,coarse,theta", [((1, 1, 300), 8, 16, 0.05), ((9, 7, 5), 8, 100, 0.05),
                                                       ((33, 27, 19), 8, 16, 0.05), ((33, 27, 19), 3, 16, 0.05),
                                                       ((33, 27, 19), 2, 16, 0.05), ((64, 57, 12), 8, 450, 0.05),
                                                       ((64, 57, 17), 8, 16, 0.0), ((64, 57, 22), 8, 128, 0.0)], ids=str)
def test_cycle_tail(shape, nlevel, coarse, theta, sweeps):
    from msg123_b200.solver import GpuSolver
    kw = dict(precon_type=1, ref_quirks=0, amg_coarse_max=coarse, amg_nlevel=nlevel, amg_sweeps=sweeps, amg_theta=theta)
    p = make_config("hetero", shape=shape, seed=7)
    o = Oracle(p, **kw)
    o.init_state()
    o.set_state(head_new=p.head0 + 0.004 * np.random.default_rng(3).standard_normal(p.ncalc), delt=3600.0)
    d, lu, r = o.make_matvec()
    o.set_system(d, lu, r)
    v = np.random.default_rng(5).standard_normal(p.ncalc)
    zo = o.precond(v)
    with GpuSolver(p, **kw) as g:
        g.set_system(d, lu, r)
        assert np.array_equal(g.precond(v), zo)
        assert np.array_equal(g.precond(v), zo)
    with GpuSolver(p, precision=1, **kw) as g:
        g.set_system(d, lu, r)
        assert np.linalg.norm(g.precond(v) - zo) <= 2e-2 * np.linalg.norm(zo)
    o.close()
