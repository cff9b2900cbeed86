"""Rows in slabs (irwls_debug_slab_bytes): the plain Gram and the tensor-core predictions on data
that in earnest only many GB reach, against the references of their own tests."""
import ctypes as C

import numpy as np
import pytest

import test_gpu_gram_plain as gram
import test_gpu_predict_tc as predict
from libirwls_gb300 import load

pytestmark = pytest.mark.gpu


@pytest.fixture
def slab():
    f = load().irwls_debug_slab_bytes
    f.argtypes, f.restype = [C.c_size_t], None
    yield f
    f(0)


# a 16-row block of two 128-column tiles is 56 KB: slabs of one block, of several with a rest, of all rows
@pytest.mark.parametrize("l,m,nact,blocks,P", [(200, 128, 200, 1, 13), (700, 200, 613, 7, 20), (3000, 130, 2500, 50, 9),
                                               (300, 128, 290, 30, 2)])
def test_gram(slab, l, m, nact, blocks, P):
    slab(blocks * 2 * 7 * 128 * 16 * 2)
    lib = load()
    lib.irwls_par_gram_min_parts.argtypes = [C.c_int, C.c_int]
    assert lib.irwls_par_gram_min_parts(l, m) == -(-l // (16 * blocks)) <= P
    gram.test_against_exact_products(l, m, nact, P)


# a 128-row tile of 16 features is 28 KB: slabs of one tile and of several with a rest; one and several drains
@pytest.mark.parametrize("kind,n,d,nsv,gamma,tiles", [("onehot", 1300, 16, 400, 0.1, 1), ("dense", 4001, 17, 130, 0.4, 3),
                                                      ("dense", 1500, 300, 700, 0.4, 2)])
def test_predictions(slab, kind, n, d, nsv, gamma, tiles):
    slab(tiles * -(-d // 16) * 28672)
    predict.test_against_extended_precision(kind, n, d, nsv, gamma)
