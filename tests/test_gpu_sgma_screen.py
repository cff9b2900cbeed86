"""The plain form's SGMA through the screened selection (tensor-core scores
with a measured error bound, FP64 scores for the steps they do not settle):
the centroids must be those of the FP64 scores, which verbose = 1 asks for at
every step, and the CPU restatement's."""
import numpy as np
import pytest

import harness as H
from libirwls_gb300 import _abi, load, synth

pytestmark = pytest.mark.gpu


def _data(kind, n, seed):
    if kind == "onehot":
        return synth.mixed_onehot(n, seed)
    X, y = synth.two_gaussians(n, 7, seed)
    if kind == "repeated":  # every row three times: exact ties between different rows
        X, y = np.repeat(X[:n // 3], 3, axis=0), np.repeat(y[:n // 3], 3)
    if kind == "few":  # fewer distinct rows than centroids: residuals and pivots vanish
        X, y = np.tile(X[:24], (n // 24, 1)), np.tile(y[:24], n // 24)
    if kind == "far":  # kernel values near zero
        X = X * 40.0
    return synth.from_dense(X, y, keep_zeros=kind != "sparse")


def _sgma(lib, hd, m, gamma, verbose):
    p = _abi.make_properties(gamma=gamma, C_=10.0, size=m, algorithm=1, verbose=verbose)
    lib.initMemory(1, m)
    H.LIBC.srand(5)
    return H.arr(lib.SGMA(hd.struct, p), m, np.int32)


# one row tile and its edges, several; orders around the 32-column stages
@pytest.mark.parametrize("kind,n,m,gamma", [("onehot", 127, 20, 0.1), ("onehot", 1500, 66, 0.1), ("dense", 129, 33, 0.2),
                                            ("sparse", 800, 31, 0.05), ("repeated", 900, 40, 0.2), ("far", 400, 24, 0.1)])
def test_centroids_of_the_fp64_scores(kind, n, m, gamma):
    s = _data(kind, n, n + m)
    hd = _abi.build_dataset(s.indptr, s.indices, s.values, s.y)
    got = _sgma(load(), hd, m, gamma, 0)
    assert np.array_equal(got, _sgma(load(), hd, m, gamma, 1))
    assert np.array_equal(got, _sgma(H.port(), hd, m, gamma, 0))


def test_budget_beyond_the_rank():
    s = _data("few", 480, 3)
    hd = _abi.build_dataset(s.indptr, s.indices, s.values, s.y)
    assert np.array_equal(_sgma(load(), hd, 40, 0.3, 0), _sgma(load(), hd, 40, 0.3, 1))
