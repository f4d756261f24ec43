"""A call that fails on the host's side or gives up a bounded wait leaves a context that works:
the next call gives the bits of the oracle."""
import numpy as np
import pytest

from msg123_b200 import abi
from msg123_b200.config import make_config
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def _system(shape, **kw):
    """Problem, system at a perturbed head, and the oracle that holds it."""
    p = make_config("hetero", shape=shape, seed=4, **kw)
    o = Oracle(p)
    o.init_state()
    o.set_state(head_new=p.head0 + 0.01 * np.random.default_rng(7).standard_normal(p.ncalc))
    sys = o.make_matvec()
    o.set_system(*sys)
    return p, o, sys


@pytest.mark.parametrize("sweep", [1, 2, 3])
def test_refused_sweep_launch(sweep):
    """A DILU sweep (factor, forward, backward) whose launch is refused: the following sweeps
    take their tiles from the start of the order again."""
    from msg123_b200.solver import GpuSolver, MsgError
    p, o, sys = _system((40, 20, 5), precon_type=0)
    v = np.random.default_rng(1).standard_normal(p.ncalc)
    with GpuSolver(p) as g:
        g.set_system(*sys)
        g.test_hook(abi.HOOK_SWEEP_LAUNCH, sweep)
        with pytest.raises(MsgError, match="launch"):
            g.precond(v)
        for _ in range(2):
            assert np.array_equal(g.precond(v), o.precond(v))
    o.close()


@pytest.mark.parametrize("shape,tile", [((40, 20, 5), 1), ((40, 20, 5), 5), ((33, 25, 2), 4)], ids=str)
def test_wait_between_tiles_runs_out(shape, tile):
    """A tile that hands nothing over: the call reports the wait that ran out, through the
    preconditioner and through the solver (whose host waits look at another word), and the same
    context goes on with right values."""
    from msg123_b200.solver import GpuSolver, MsgError
    p, o, sys = _system(shape, precon_type=0)
    v = np.random.default_rng(1).standard_normal(p.ncalc)
    with GpuSolver(p) as g:
        g.set_system(*sys)
        good = g.solve_linalg(float(sys[2] @ sys[2]), 1e-8, np.zeros(p.ncalc))
        for _ in range(2):
            g.test_hook(abi.HOOK_SWEEP_WITHHOLD, tile)
            with pytest.raises(MsgError, match="wait between tiles"):
                g.precond(v)
            assert np.array_equal(g.precond(v), o.precond(v))
        g.test_hook(abi.HOOK_SWEEP_WITHHOLD, tile)
        with pytest.raises(MsgError, match="wait between tiles"):
            g.solve_linalg(float(sys[2] @ sys[2]), 1e-8, np.zeros(p.ncalc))
        again = g.solve_linalg(float(sys[2] @ sys[2]), 1e-8, np.zeros(p.ncalc))
        assert all(np.array_equal(a, b) for a, b in zip(good, again))
    o.close()


def _pool_bytes():
    """Bytes handed out by the device's default memory pool (cudaMemPoolAttrUsedMemCurrent)."""
    import ctypes as C
    from msg123_b200.solver import load_library
    load_library()
    rt, pool, used = C.CDLL("libcudart.so.12"), C.c_void_p(), C.c_uint64()
    assert rt.cudaDeviceSynchronize() == 0
    assert rt.cudaDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    assert rt.cudaMemPoolGetAttribute(pool, 7, C.byref(used)) == 0
    return used.value


@pytest.mark.parametrize("precision,coarse", [(0, 16), (1, 16), (0, 200)])
def test_failed_hierarchy_build(precision, coarse):
    """No memory at any of a build's allocations: set_system fails, the preconditioner refuses to
    run on what there is, nothing stays allocated, and the next call of a run that would keep its
    hierarchy for several steps (amg_lag) builds one.  (Without memory for the places of a
    product the build goes on with exact ones: the same bits.)"""
    from msg123_b200.solver import GpuSolver, MsgError
    kw = dict(precon_type=1, ref_quirks=0, amg_coarse_max=coarse, amg_lag=8)
    p, o, sys = _system((33, 27, 19))
    v = np.random.default_rng(1).standard_normal(p.ncalc)
    with GpuSolver(p, precision=precision, **kw) as ref:
        ref.set_system(*sys)
        want = ref.precond(v)
    if precision == 0:
        oa = Oracle(p, **kw)
        oa.set_system(*sys)
        assert np.array_equal(want, oa.precond(v))
        oa.close()
    before = _pool_bytes()
    with GpuSolver(p, precision=precision, **kw) as g:
        g.init_state()
        g.set_system(*sys)
        empty, failed = None, 0
        for k in range(1, 120):
            g.test_hook(abi.HOOK_AMG_ALLOC, k)
            try:
                g.set_system(*sys)
            except MsgError as e:
                assert "memory" in str(e)
            else:
                assert np.array_equal(g.precond(v), want)
                continue
            failed += 1
            with pytest.raises(MsgError, match="not built"):
                g.precond(v)
            empty = empty or _pool_bytes()
            assert _pool_bytes() == empty, k
        assert failed > 60
        g.test_hook(abi.HOOK_AMG_ALLOC, 0)
        g.set_system(*sys)
        assert np.array_equal(g.precond(v), want)
        # a step after a build that failed: the hierarchy is built again, lag or not
        g.test_hook(abi.HOOK_AMG_ALLOC, 30)
        with pytest.raises(MsgError):
            g.set_system(*sys)
        g.calc_numsol()
        assert g.amg_levels()[1]["n"] > 1
    assert _pool_bytes() == before
    o.close()
