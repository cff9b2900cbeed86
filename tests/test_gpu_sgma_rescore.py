"""The screened selection's FP64 scores of the candidates that can be the best:
rows repeated so that two to many candidates tie, at sizes around the 64-row and
8-column steps of the kernel for up to four of them and the 16-candidate groups of
the other; the centroids must be those of all candidates' FP64 scores (verbose = 1)
and the CPU restatement's."""
import numpy as np
import pytest

import harness as H
from libirwls_gb300 import _abi, load, synth

pytestmark = pytest.mark.gpu


def _sgma(lib, hd, m, verbose):
    p = _abi.make_properties(gamma=0.2, C_=10.0, size=m, algorithm=1, verbose=verbose)
    lib.initMemory(1, m)
    H.LIBC.srand(7)
    return H.arr(lib.SGMA(hd.struct, p), m, np.int32)


# distinct rows, rows, budget: about 2, 5, 16 and more than 30 copies of the best among the 64 candidates
@pytest.mark.parametrize("distinct,n,m", [(400, 801, 41), (60, 500, 19), (20, 640, 9), (4, 129, 3)])
def test_tied_candidates(distinct, n, m):
    X, y = synth.two_gaussians(distinct, 7, n)
    reps = -(-n // distinct)
    s = synth.from_dense(np.tile(X, (reps, 1))[:n], np.tile(y, reps)[:n], keep_zeros=True)
    hd = _abi.build_dataset(s.indptr, s.indices, s.values, s.y)
    got = _sgma(load(), hd, m, 0)
    assert np.array_equal(got, _sgma(load(), hd, m, 1))
    assert np.array_equal(got, _sgma(H.port(), hd, m, 0))
