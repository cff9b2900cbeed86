"""A row's decision value does not depend on the rows beside it: the same bits from any split
of a batch below 500000 kernel values (more rows per CTA from 608 rows on). Above, the sums are
the tensor-core path's, within the rounding of both (its digits within 2^-56 of a row's scale
per feature, its exponent within 4 units of 2^-56, a value's two roundings and the sum's)."""
import ctypes as C

import numpy as np
import pytest

from libirwls_gb300 import _abi, load

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def _set(M):
    n, d = M.shape
    r, c = np.nonzero(M)
    return _abi.build_dataset(np.r_[0, np.cumsum(np.bincount(r, minlength=n))], c + 1, M[r, c], np.ones(n), False)


def _soft(M, mdl):
    T = _set(M)
    f = load().softTest(T.struct, mdl, _abi.make_predict_properties())
    return np.ctypeslib.as_array(f, shape=(len(M),)).copy()


@pytest.mark.parametrize("n,d,nsv,kernel", [(3000, 7, 130, 1), (1300, 20, 300, 1), (2600, 5, 33, 0), (9000, 900, 40, 1)])
def test_splits(n, d, nsv, kernel):
    rng = np.random.default_rng(n)
    A, B = rng.standard_normal((n, d)), rng.standard_normal((nsv, d))
    A[rng.random(A.shape) < 0.5] = 0.0
    w, S = rng.standard_normal(nsv), _set(B)
    mdl = load().calculateFULLModel(_abi.make_properties(gamma=1.0 / d, kernel=kernel), S.struct,
                                    np.r_[w, 0.1].ctypes.data_as(C.POINTER(C.c_double)))
    whole = _soft(A, mdl)
    pick = [0, 1, n - 1]
    assert np.array_equal(np.concatenate([_soft(A[i:i + 1], mdl) for i in pick]), whole[pick])
    for k in (300, 700, 1999):
        assert np.array_equal(np.concatenate([_soft(A[i:i + k], mdl) for i in range(0, n, k)]), whole)


def test_across_the_paths():
    n, d, nsv, gamma = 4000, 20, 300, 0.05
    rng = np.random.default_rng(1)
    A, B, w = rng.standard_normal((n, d)), rng.standard_normal((nsv, d)), rng.standard_normal(nsv)
    S = _set(B)
    mdl = load().calculateFULLModel(_abi.make_properties(gamma=gamma), S.struct,
                                    np.r_[w, 0.1].ctypes.data_as(C.POINTER(C.c_double)))
    whole, parts = _soft(A, mdl), np.concatenate([_soft(A[i:i + 1000], mdl) for i in range(0, n, 1000)])
    qa, qb = (A * A).sum(1), (B * B).sum(1)
    k = np.exp(-gamma * (qa[:, None] + qb - 2 * A @ B.T))
    rel = gamma * (2 * d * 2.1 ** 2 * np.sqrt(qa[:, None] * qb) * 2.0 ** -55 + (d + 4) * EPS * (qa[:, None] + qb)) + 8 * EPS
    assert np.all(np.abs(whole - parts) <= (np.abs(w) * k * rel).sum(1) + 2 * (nsv + 64) * EPS * ((np.abs(w) * k).sum(1) + 0.1))
