"""Small levels of a V-cycle in one cluster launch against the same levels by a launch per pass, bit
for bit in FP64 and in the mixed cycle: a row's sum runs in the same order in both.  (Against the
FP64 oracle the mixed cycle's bound does not see the small levels: they are a hundredth of z.)"""
import numpy as np
import pytest

from msg123_b200 import abi
from msg123_b200.config import make_config
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sweeps", [0, 1, 2, 3])
@pytest.mark.parametrize("shape,nlevel,coarse,theta", [((1, 1, 300), 8, 16, 0.05), ((9, 7, 5), 8, 100, 0.05),
                                                       ((33, 27, 19), 8, 16, 0.05), ((33, 27, 19), 3, 16, 0.05),
                                                       ((33, 27, 19), 2, 16, 0.05), ((64, 57, 12), 8, 450, 0.05),
                                                       ((64, 57, 17), 8, 16, 0.0), ((64, 57, 22), 8, 128, 0.0),
                                                       ((113, 87, 37), 8, 128, 0.05)], ids=str)
def test_cycle_tail_bits(shape, nlevel, coarse, theta, sweeps):
    from msg123_b200.solver import GpuSolver, launch_count
    kw = dict(precon_type=1, ref_quirks=0, amg_coarse_max=coarse, amg_nlevel=nlevel, amg_sweeps=sweeps, amg_theta=theta)
    p = make_config("hetero", shape=shape, seed=7)
    o = Oracle(p, **kw)
    o.init_state()
    o.set_state(head_new=p.head0 + 0.004 * np.random.default_rng(3).standard_normal(p.ncalc), delt=3600.0)
    system = o.make_matvec()
    o.close()
    v = np.random.default_rng(5).standard_normal(p.ncalc)
    for precision in (0, 1):
        with GpuSolver(p, precision=precision, **kw) as g:
            g.set_system(*system)
            got, launches = [], []
            for off in (0, 1, 0):
                g.test_hook(abi.HOOK_CYCLE_LAUNCHES, off)
                n = launch_count()
                got.append(g.precond(v))
                launches.append(launch_count() - n)
            assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
            small = g.amg_levels()[1:]
            dense = small[-1]["n"] <= coarse
            # a last level of more than 512 rows keeps the launches; a dense level, or one of a
            # single pass, is one launch either way
            if small[-1]["n"] <= 512 and (len(small) > 1 or (not dense and sweeps > 1)):
                assert launches[0] < launches[1] and launches[2] == launches[0]
            else:
                assert launches[0] == launches[1]
