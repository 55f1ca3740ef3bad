"""fg_host_free on each kind of memory that it frees: fg_host_alloc's, the
columns of fg_pattern_build, and those after the caller page-locked them (the
registration has to go with them), small and of several huge pages."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Attributes(C.Structure):  # cudaPointerAttributes
    _fields_ = [("type", C.c_int), ("device", C.c_int), ("device_pointer", C.c_void_p), ("host_pointer", C.c_void_p),
                ("reserved", C.c_long * 8)]


def memory_type(ptr):
    a = Attributes()
    with open("/proc/self/maps") as f:
        path = next(line.split()[-1] for line in f if "libcudart.so" in line)
    assert C.CDLL(path).cudaPointerGetAttributes(C.byref(a), C.c_void_p(ptr)) == 0
    return a.type


UNREGISTERED, HOST = 0, 1


def columns(femg, m):
    prob = femg.Problem(femg.config_c2(m=m, order=2))
    a = prob.arrays()
    edof, etype = np.ascontiguousarray(a["edof"]), np.ascontiguousarray(a["etype"])
    ai, aj = np.zeros(int(a["n_rows"]) + 1, np.uint64), C.c_void_p()
    femg.check(femg.lib().fg_pattern_build(edof.ctypes.data, etype.ctypes.data, edof.shape[0], edof.shape[1], int(a["n_rows"]),
                                           ai.ctypes.data, C.byref(aj), 0, None, 0))
    assert np.array_equal(ai, a["ai"])
    return aj.value, int(ai[-1]) * 8


@pytest.mark.parametrize("m", [1, 12])
@pytest.mark.parametrize("registered", [False, True])
def test_pattern_columns(femg, cuda, registered, m):
    cudart = cuda.cuda.cudart()
    ptr, size = columns(femg, m)
    assert memory_type(ptr) == UNREGISTERED
    if registered:
        assert int(cudart.cudaHostRegister(ptr, size, 0)) == 0
        assert memory_type(ptr) == HOST
    femg.lib().fg_host_free(ptr)
    assert memory_type(ptr) == UNREGISTERED


def test_page_locked_buffer(femg, cuda):
    cuda.zeros(1, device="cuda")
    p = C.c_void_p()
    femg.check(femg.lib().fg_host_alloc(C.byref(p), 1 << 20))
    assert memory_type(p.value) == HOST
    femg.lib().fg_host_free(p)
    assert memory_type(p.value) == UNREGISTERED
    femg.lib().fg_host_free(None)
