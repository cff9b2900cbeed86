"""Full training and subIRWLS without room for the kept kernel matrix: each iteration forms its
kernel values, and the weights are the same up to rounding."""
import ctypes as C

import numpy as np
import pytest

import harness as H
from libirwls_gb300 import _abi, load, synth

pytestmark = pytest.mark.gpu
PD = C.POINTER(C.c_double)


@pytest.fixture
def lib():
    lib = load()
    lib.irwls_debug_alloc_limit.argtypes, lib.irwls_debug_alloc_limit.restype = [C.c_size_t], None
    yield lib
    lib.irwls_debug_alloc_limit(0)


# K takes (w + 6)^2 doubles, the system (w + 2)^2: limits between the two
@pytest.mark.parametrize("n,w,dense", [(300, 100, True), (900, 350, False)])
def test_training(lib, n, w, dense):
    X, y = synth.two_gaussians(n, 5, n, shift=0.9)
    s = synth.from_dense(X, y, keep_zeros=dense)
    hd = _abi.build_dataset(s.indptr, s.indices, s.values, s.y)
    p = dict(gamma=0.3, C=10.0, kernel=1, w=w)
    kept = H.run_full(lib, hd, p)[0]
    lib.irwls_debug_alloc_limit(8 * (w + 2) ** 2)
    direct = H.run_full(lib, hd, p)[0]
    assert lib.irwls_last_error() == 0
    assert np.array_equal(kept[:-1] != 0, direct[:-1] != 0)
    assert H.rel_err(direct, kept) <= H.REL_TOL


def test_sub(lib):
    n = 200
    X, y = synth.two_gaussians(n, 5, 1, shift=0.9)
    s = synth.from_dense(X, y, keep_zeros=True)
    hd = _abi.build_dataset(s.indptr, s.indices, s.values, s.y)
    lib.subIRWLS.restype = PD
    out = []
    for limit in (0, 8 * (n + 2) ** 2):
        lib.irwls_debug_alloc_limit(limit)
        GIN, e, beta = np.zeros(n + 1), y.astype(float).copy(), np.zeros(n + 1)
        prop = _abi.make_properties(gamma=0.3, C_=10.0, working_set=n)
        lib.subIRWLS.argtypes = [type(hd.struct), type(prop), PD, PD, PD]
        out.append(H.arr(lib.subIRWLS(hd.struct, prop, *[a.ctypes.data_as(PD) for a in (GIN, e, beta)]), n + 1))
    assert H.rel_err(out[1], out[0]) <= H.REL_TOL
