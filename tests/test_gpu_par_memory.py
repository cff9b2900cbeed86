"""IRWLSpar of 128 centroids and more where memory is short: without the digits' workspace the
FP64 Gram serves (its products against extended precision as those of small budgets), and the
weights are the reference's either way."""
import ctypes as C

import numpy as np
import pytest

import harness as H
import test_gpu_gram_fp64 as small
from libirwls_gb300 import _abi, load, synth

pytestmark = pytest.mark.gpu


# the edges of the 64 x 64 tiles, the row of the right-hand side in a tile of its own, chunks without a row
@pytest.mark.parametrize("l,m,nact,P", [(300, 128, 290, 2), (200, 129, 7, 3), (400, 191, 333, 5), (700, 300, 700, 1)])
def test_wide_products(l, m, nact, P):
    small.test_against_exact_products(l, m, nact, P)


# what each limit refuses: the slices (7 MB), the slices of a larger set; K_nm takes 2.2 and 8 MB
@pytest.mark.parametrize("l,m,limit", [(2000, 140, 4 << 20), (4000, 260, 10 << 20)])
def test_training(l, m, limit):
    lib = load()
    lib.irwls_debug_alloc_limit.argtypes, lib.irwls_debug_alloc_limit.restype = [C.c_size_t], None
    s = synth.mixed_onehot(l, m)
    hd = _abi.build_dataset(s.indptr, s.indices, s.values, s.y)
    p = dict(gamma=0.1, C=10.0, kernel=1, size=m, algorithm=0)
    cent, want, _, _, _ = H.run_budget(H.port(), hd, p)
    plain = H.run_budget(lib, hd, p)[1]
    lib.irwls_debug_alloc_limit(limit)
    try:
        got = H.run_budget(lib, hd, p)
        assert lib.irwls_last_error() == 0
    finally:
        lib.irwls_debug_alloc_limit(0)
    assert np.array_equal(got[0], cent) and not np.array_equal(got[1], plain)
    assert H.rel_err(got[1], want) <= H.REL_TOL and H.rel_err(plain, want) <= H.REL_TOL
