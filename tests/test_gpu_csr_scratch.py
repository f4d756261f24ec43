"""The Jacobian in CSR order through the vectors of a solve: out as the oracle's bits and in again
(the preconditioner of the system set equals the assembled one's), on grids of a few cells and
of lengths between the vectors' boundaries, and no device memory kept by either call."""
import ctypes as C

import numpy as np
import pytest

from msg123_b200.config import make_config
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def _free_bytes():
    rt, free, total = C.CDLL("libcudart.so.12"), C.c_size_t(), C.c_size_t()
    assert rt.cudaDeviceSynchronize() == 0 and rt.cudaMemGetInfo(C.byref(free), C.byref(total)) == 0
    return free.value


@pytest.mark.parametrize("shape", [(1, 1, 2), (1, 7, 1), (9, 1, 1), (3, 4, 5), (29, 29, 1), (10, 10, 9), (1, 60, 41), (37, 23, 11),
                                   (2, 3, 997)], ids=str)
def test_csr_through_solve_vectors(shape):
    from msg123_b200.solver import GpuSolver
    p = make_config("hetero", shape=shape, seed=6, precon_type=0)
    rng = np.random.default_rng(3)
    h = p.head0 + 0.01 * rng.standard_normal(p.ncalc)
    o = Oracle(p)
    o.init_state()
    o.set_state(head_new=h, delt=3600.0)
    with GpuSolver(p) as g:
        g.init_state()
        g.set_state(head_new=h, delt=3600.0)
        for got, want in zip(g.make_matvec(), o.make_matvec()):
            # the van Genuchten pow differs by rounding
            assert np.max(np.abs(got - want), initial=0.0) <= 1e-8 * np.max(np.abs(want), initial=0.0)
        d, lu, r = g.make_matvec()
        v = rng.standard_normal(p.ncalc)
        z = g.precond(v)
        g.set_system(2.0 * d, 2.0 * lu, 2.0 * r)
        assert np.array_equal(g.precond(2.0 * v), z)
        o.set_system(d, lu, r)
        assert np.array_equal(z, o.precond(v))
    o.close()


def test_csr_calls_keep_no_memory():
    from msg123_b200.solver import GpuSolver
    p = make_config("hetero", shape=(160, 160, 48), seed=6, precon_type=0)
    with GpuSolver(p) as g:
        g.init_state()
        g.make_matvec()                       # the copy pool and the kernels' own memory
        with GpuSolver(p) as fresh:
            fresh.init_state()
            before = _free_bytes()
            d, lu, r = fresh.make_matvec()
            fresh.set_system(d, lu, r)
            assert before - _free_bytes() < lu.nbytes // 2
