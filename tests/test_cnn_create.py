"""A network that cannot be made (no GPU here) gives back what it had taken."""
import ctypes as C

import pytest

from msg123_b200.solver import load_library


class _MallInfo(C.Structure):
    _fields_ = [(f, C.c_size_t) for f in ("arena", "ordblks", "smblks", "hblks", "hblkhd", "usmblks", "fsmblks", "uordblks",
                                          "fordblks", "keepcost")]


def test_failed_create_keeps_nothing():
    import torch
    if torch.cuda.is_available():
        pytest.skip("the call succeeds on a GPU")
    L, libc = load_library(), C.CDLL(None)
    libc.mallinfo2.restype = _MallInfo
    L.msg_gpu_cnn_create.argtypes = [C.c_int32, C.POINTER(C.c_void_p)]
    h = C.c_void_p()
    for _ in range(100):
        assert L.msg_gpu_cnn_create(1, C.byref(h)) < 0 and not h.value
    before = libc.mallinfo2().uordblks
    for _ in range(2000):
        L.msg_gpu_cnn_create(1, C.byref(h))
    assert libc.mallinfo2().uordblks - before < 100_000
