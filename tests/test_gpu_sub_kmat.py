"""The inner loop of full IRWLS on the working set's kept kernel matrix (sets
up to 4096 rows) and without it, against the CPU restatement: sets around the
512-thread bookkeeping kernels' size, a set larger than the training set, and
one above the kept size."""
import numpy as np
import pytest

import harness as H
from libirwls_gb300 import _abi, load, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,w,dense,cost", [(300, 3, 7, True, 1.0), (900, 5, 33, False, 10.0), (1200, 4, 511, True, 10.0),
                                              (1200, 4, 512, False, 10.0), (1100, 4, 700, True, 1.0),
                                              (200, 4, 500, True, 10.0), (4300, 3, 4200, True, 0.05)])
def test_training_matches_the_restatement(n, d, w, dense, cost):
    X, y = synth.two_gaussians(n, d, 100 + n + w, shift=0.9)
    s = synth.from_dense(X, y, keep_zeros=dense)
    hd = _abi.build_dataset(s.indptr, s.indices, s.values, s.y)
    p = dict(gamma=0.3, C=cost, kernel=1, w=w)
    got, _, _ = H.run_full(load(), hd, p)
    ref, _, _ = H.run_full(H.port(), hd, p)
    assert np.array_equal(got[:-1] != 0, ref[:-1] != 0)
    assert H.rel_err(got, ref) <= H.REL_TOL
