"""Hierarchy build on the GPU against the oracle, bit for bit, where the build's passes change
form: columns and single layers, tile remainders, every strength threshold from all
neighbours strong (long prolongation and product rows, columns beyond the register and short
table sizes) to few, levels on both sides of the one-cluster aggregation."""
import numpy as np
import pytest

from msg123_b200.config import make_config
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,theta,delt", [((1, 1, 300), 0.05, 3600.0), ((33, 9, 2), 0.05, 3600.0),
                                              ((70, 1, 5), 0.05, 600.0), ((48, 40, 24), 0.0, 3600.0),
                                              ((48, 40, 24), 0.3, 3600.0), ((37, 29, 31), 0.0, 60.0),
                                              ((96, 80, 40), 0.05, 36000.0), ((96, 80, 40), 0.0, 3600.0)], ids=str)
def test_hierarchy_forms_bitexact(shape, theta, delt):
    from msg123_b200.solver import GpuSolver
    kw = dict(precon_type=1, ref_quirks=0, amg_coarse_max=16, amg_theta=theta)
    p = make_config("hetero", shape=shape, seed=5)
    o = Oracle(p, **kw)
    o.init_state()
    o.set_state(head_new=p.head0 + 0.02 * np.random.default_rng(1).standard_normal(p.ncalc), delt=delt)
    d, lu, r = o.make_matvec()
    o.set_system(d, lu, r)
    with GpuSolver(p, **kw) as g:
        g.set_system(d, lu, r)
        lg, lo = g.amg_levels(), o.amg_levels()
        assert len(lg) == len(lo)
        for a, b in zip(lg, lo):
            assert a["n"] == b["n"]
            for k in ("offind", "offrow", "dmat", "lumat", "pindex", "poffrow", "pval", "agg"):
                if k in a:
                    assert np.array_equal(a[k], b[k]), k
        v = np.random.default_rng(2).standard_normal(p.ncalc)
        assert np.array_equal(g.precond(v), o.precond(v))
    o.close()
