"""More separate summed indices than a mode group holds are refused: A and B of rank eight with no
index in common, all summed (the Python front end's semantics), in orders that do not merge."""
import ctypes

import pytest


@pytest.fixture(scope="module")
def lib():
    from einsums_gb300 import _lib, build
    build.build()
    return _lib.load()


def test_sixteen_summed_indices(lib):
    from einsums_gb300 import _lib
    T = _lib.EgTensor
    C, A, B = T(), T(), T()
    C.rank = 0
    C.data = 16
    for t in (A, B):
        t.rank, t.data = 8, 16
        for d in range(8):
            t.extent[d], t.stride[d] = 2, 3 ** d  # no two modes are one
    opt = _lib.EgOptions(0, 0, 1e-10, 1, 0)  # Python semantics
    st = lib.eg_einsum(0.0, _lib.labels(""), ctypes.byref(C), 1.0, _lib.labels("abcdefgh"), ctypes.byref(A),
                       _lib.labels("ijklmnop"), ctypes.byref(B), ctypes.byref(opt), None, None)
    assert st == 4
    assert b"separate indices" in lib.eg_last_error()
