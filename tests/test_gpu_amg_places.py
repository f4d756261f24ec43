"""Hierarchy products whose places are not of the products' size (as beyond 32-bit offsets or the
memory) but found by a first pass over the rows: bit for bit the oracle's hierarchy, with rows
beyond the register columns of the fine level (every neighbour strong), the short table and the
middle one.  And the scan that tells: its total in 64 bits."""
import numpy as np
import pytest

from msg123_b200 import abi
from msg123_b200.config import make_config
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("most", [1, 20000])
@pytest.mark.parametrize("shape,theta,delt", [((1, 1, 300), 0.05, 3600.0), ((33, 9, 2), 0.05, 3600.0),
                                              ((37, 29, 31), 0.0, 60.0), ((48, 40, 24), 0.05, 36000.0)], ids=str)
def test_places_from_row_lengths(shape, theta, delt, most):
    from msg123_b200.solver import GpuSolver
    kw = dict(precon_type=1, ref_quirks=0, amg_coarse_max=16, amg_theta=theta)
    p = make_config("hetero", shape=shape, seed=5)
    o = Oracle(p, **kw)
    o.init_state()
    o.set_state(head_new=p.head0 + 0.02 * np.random.default_rng(1).standard_normal(p.ncalc), delt=delt)
    d, lu, r = o.make_matvec()
    o.set_system(d, lu, r)
    with GpuSolver(p, **kw) as g:
        g.test_hook(abi.HOOK_AMG_PRODUCTS, most)
        g.set_system(d, lu, r)
        lg, lo = g.amg_levels(), o.amg_levels()
        assert len(lg) == len(lo)
        for a, b in zip(lg, lo):
            for k in ("offind", "offrow", "dmat", "lumat", "pindex", "poffrow", "pval", "agg"):
                if k in a:
                    assert np.array_equal(a[k], b[k]), k
    o.close()


@pytest.mark.parametrize("n,top", [(1, 9), (4095, 30), (4096, 30), (4097, 30), (60000, 30), (4097, 1 << 20), (60000, 1 << 20)])
def test_scan_total(n, top):
    from msg123_b200.solver import GpuSolver
    counts = np.random.default_rng(n).integers(0, top, n)
    with GpuSolver(make_config("hetero", shape=(60, 50, 20), seed=1)) as g:
        out, total = g.scan(counts)
    sums = np.concatenate([[0], np.cumsum(counts)])
    assert total == sums[-1]
    assert np.array_equal(out, sums.astype(np.uint64).astype(np.uint32).view(np.int32))
