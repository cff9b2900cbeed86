"""SGMA where memory is short: the plain form takes the FP64 scores of all candidates, which
need K_nm alone, and the same candidates; with room for the screening but not for the rows
ahead, the explicit inverse serves, in both forms."""
import ctypes as C

import numpy as np
import pytest

import harness as H
from libirwls_gb300 import _abi, load, synth

pytestmark = pytest.mark.gpu
PI, PD = C.POINTER(C.c_int), C.POINTER(C.c_double)
L, M = 1500, 66


@pytest.fixture
def lib():
    lib = load()
    assert lib.irwls_gpu_available(), lib.irwls_last_error_message()
    lib.irwls_debug_fail_alloc.argtypes, lib.irwls_debug_fail_alloc.restype = [C.c_longlong], None
    lib.irwls_debug_alloc_limit.argtypes, lib.irwls_debug_alloc_limit.restype = [C.c_size_t], None
    yield lib
    lib.irwls_debug_fail_alloc(0)
    lib.irwls_debug_alloc_limit(0)
    lib.irwls_set_precision(0)


@pytest.fixture
def resident(lib):
    s = synth.mixed_onehot(L, 7)
    hd = _abi.build_dataset(s.indptr, s.indices, s.values, s.y)
    props = _abi.make_properties(gamma=0.1, C_=10.0, size=M, algorithm=1)
    h = lib.irwls_resident_upload(hd.struct, props, 1)
    assert h
    yield lambda: _train(lib, h, props)
    lib.irwls_resident_free(h)


def _train(lib, h, props):
    c, w = np.zeros(M, np.int32), np.zeros(M)
    H.LIBC.srand(3)
    rc = lib.irwls_resident_budgeted(h, props, c.ctypes.data_as(PI), w.ctypes.data_as(PD))
    return rc, c, w


@pytest.mark.parametrize("k", range(1, 22))
def test_any_allocation_of_the_screening(lib, resident, k):
    rc, c0, w0 = resident()
    assert rc == 0
    lib.irwls_debug_fail_alloc(k)
    rc, c, w = resident()
    lib.irwls_debug_fail_alloc(0)
    assert rc == 0 and lib.irwls_last_error() == 0, lib.irwls_last_error_message()
    assert np.array_equal(c, c0) and np.array_equal(w, w0)


# the rows ahead take 64 m (8 m + 6 x 128) = 5.5 MB here, K_nm 0.8, Q 1.2, the
# precision form's Gram 2.7
@pytest.mark.parametrize("limit,mixed", [(4 << 20, 0), (4 << 20, 1), (1 << 20, 0)])
def test_limits(lib, resident, limit, mixed):
    lib.irwls_set_precision(mixed)
    rc, c0, _ = resident()
    assert rc == 0
    lib.irwls_debug_alloc_limit(limit)
    rc, c, _ = resident()
    lib.irwls_debug_alloc_limit(0)
    assert rc == 0 and lib.irwls_last_error() == 0, lib.irwls_last_error_message()
    assert np.array_equal(c, c0)
