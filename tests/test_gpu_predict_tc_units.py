"""The fixed point that one batch or training set shares: a far row must not cost the
others their accuracy. The bound is that of FP64 sums of d features a row (d + 4 roundings
of gamma (q_i + q_j) in the exponent, two of the value, nsv + 64 of the sum)."""
import ctypes as C

import numpy as np
import pytest

from libirwls_gb300 import _abi, load

pytestmark = pytest.mark.gpu
VP, I = C.c_void_p, C.c_int
EPS = 2.0 ** -53
D, GAMMA = 20, 0.1


def _set(M):
    n, d = M.shape
    hd = _abi.build_dataset(np.arange(n + 1) * d, np.tile(np.arange(1, d + 1), n), M.ravel(), np.ones(n), False)
    hd.struct.sparse = 1  # the kernel by norms in training too
    return hd


def _rows(far, where, seed, n):
    M = np.random.default_rng(seed).standard_normal((n, D)) * 0.7
    if where:
        M[7] *= np.sqrt(far / (M[7] @ M[7]))
    return M


@pytest.mark.parametrize("far", [1e7, 4e8])
@pytest.mark.parametrize("where", ["rows", "vectors"])
def test_predictions(far, where):
    lib, n, nsv = load(), 3000, 300
    A, B = _rows(far, where == "rows", 1, n), _rows(far, where == "vectors", 2, nsv)
    w = np.random.default_rng(3).standard_normal(nsv)
    S, T = _set(B), _set(A)
    mdl = lib.calculateFULLModel(_abi.make_properties(gamma=GAMMA), S.struct,
                                 np.r_[w, 0.0].ctypes.data_as(C.POINTER(C.c_double)))
    f = lib.softTest(T.struct, mdl, _abi.make_predict_properties())
    got = np.ctypeslib.as_array(f, shape=(n,)).copy()
    L, pick = np.longdouble, np.r_[0:7, 8:60, n - 1]
    y = GAMMA * (T.q[pick, None].astype(L) + S.q[None, :nsv] - 2 * (A[pick].astype(L) @ B.astype(L).T))
    k = np.exp(-y)
    q = GAMMA * (T.q[pick, None] + S.q[None, :nsv])
    rel = (D + 4) * EPS * np.where(k > 1e-300, q, 0) + 2 * EPS
    tol = np.sum(np.abs(w) * k * rel, 1) + (nsv + 64) * EPS * np.sum(np.abs(w) * k, 1)
    assert np.all(np.abs(got[pick] - k @ w.astype(L)) <= tol)


@pytest.mark.parametrize("far,taken", [(0, True), (1e7, False)])
def test_training_rows(far, taken):
    lib, n = load(), 2000
    hd = _set(_rows(far, far > 0, 4, n))
    lib.irwls_dev_upload.argtypes = [VP, I, I, C.c_double, I, I, VP]
    lib.irwls_exact_rows_create.restype, lib.irwls_exact_rows_create.argtypes = VP, [VP, I, I]
    lib.irwls_exact_rows_free.argtypes = lib.irwls_dev_release.argtypes = [VP]
    S = (C.c_char * 256)()
    assert lib.irwls_dev_upload(C.byref(hd.struct), n, 1, GAMMA, 0, 0, S) == 0
    E = lib.irwls_exact_rows_create(S, n, 400)
    assert bool(E) == taken
    lib.irwls_exact_rows_free(E)
    lib.irwls_dev_release(S)


def test_large_norms_of_one_size_keep_the_path():
    """Rows of |x|^2 = 8100 to 8500: FP64 sums would round more coarsely than the unit."""
    lib, n = load(), 2000
    hd = _set(np.random.default_rng(5).standard_normal((n, D)) + 20.0)
    lib.irwls_dev_upload.argtypes = [VP, I, I, C.c_double, I, I, VP]
    lib.irwls_exact_rows_create.restype, lib.irwls_exact_rows_create.argtypes = VP, [VP, I, I]
    lib.irwls_exact_rows_free.argtypes = lib.irwls_dev_release.argtypes = [VP]
    S = (C.c_char * 256)()
    assert lib.irwls_dev_upload(C.byref(hd.struct), n, 1, GAMMA, 0, 0, S) == 0
    E = lib.irwls_exact_rows_create(S, n, 400)
    assert E
    lib.irwls_exact_rows_free(E)
    lib.irwls_dev_release(S)
