"""Ordered linear predictions (one rounding per stored value) against extended
precision: d fused multiply-adds per product, one rounding per weight, nsv
additions."""
import ctypes as C

import numpy as np
import pytest

import harness as H
from libirwls_gb300 import _abi, load

pytestmark = pytest.mark.gpu


# one row per CTA to eight, chunks of 128 vectors and their remainders, empty rows
@pytest.mark.parametrize("n,d,nsv", [(1, 1, 1), (5, 40, 129), (700, 33, 1501), (3000, 3, 128), (2500, 120, 257)])
def test_against_extended_precision(n, d, nsv):
    rng = np.random.default_rng(n + d)

    def rows(k):
        M = rng.standard_normal((k, d)) * 10.0 ** rng.integers(-3, 4, (1, d))
        M[rng.random(M.shape) < 0.3] = 0.0
        M[::11] = 0.0
        r, c = np.nonzero(M)
        return M, _abi.build_dataset(np.r_[0, np.cumsum(np.bincount(r, minlength=k))], c + 1, M[r, c], np.ones(k), False)

    (A, T), (B, S) = rows(n), rows(nsv)
    w, bias = rng.standard_normal(nsv), 0.5
    lib = load()
    beta = np.concatenate([w, [bias]])
    mdl = lib.calculateFULLModel(_abi.make_properties(kernel=0), S.struct,
                                 beta.ctypes.data_as(C.POINTER(C.c_double)))
    got = H.arr(lib.softTest(T.struct, mdl, _abi.make_predict_properties()), n)
    L = np.longdouble
    ref = (A.astype(L) @ B.astype(L).T) @ w.astype(L) + L(bias)
    mag = (np.abs(A) @ np.abs(B).T) @ np.abs(w) + bias
    assert np.all(np.abs(got - ref) <= (d + nsv + 2) * 2.0 ** -53 * mag)
