"""The backward sweep with its last block by substitution and by the inverse:
both solve the system with a residual of at most 8 n eps |A| |x| (each of the
factorization's and the sweeps' n-term sums rounds to n eps of its magnitudes),
and the factor is the same."""
import ctypes as C

import numpy as np
import pytest

from libirwls_gb300 import load

pytestmark = pytest.mark.gpu
VP, I = C.c_void_p, C.c_int


# one block whole and partial, the last block of one row, cluster sizes, the first order with another sweep
@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 95, 257, 1000, 2048, 2049])
def test_both_solve(n):
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n)) / np.sqrt(n)
    A, b = G @ G.T + np.eye(n), rng.standard_normal(n)
    lib = load()
    assert lib.irwls_dev_init() == 0  # (the status words that the kernels write)
    lib.irwls_dev_malloc.argtypes = [C.POINTER(VP), C.c_size_t]
    lib.irwls_dev_h2d.argtypes = lib.irwls_dev_d2h.argtypes = [VP, VP, C.c_size_t]
    lib.irwls_dev_free.argtypes = [VP]
    ld, out = n + 1, []
    for f in (lib.irwls_dev_chol_solve, lib.irwls_dev_chol_solve_order, lib.irwls_dev_chol_solve):
        f.argtypes = [VP, I, I, VP, VP]
        M = np.zeros((n, ld))
        M[:, :n] = A  # (column-major: row c holds column c)
        x, L = np.zeros(n), np.zeros((n, ld))
        bufs = []
        for a in (M, b, x):
            p = VP()
            assert lib.irwls_dev_malloc(C.byref(p), a.nbytes) == 0
            assert lib.irwls_dev_h2d(p, a.ctypes.data, a.nbytes) == 0 and lib.irwls_dev_sync() == 0
            bufs.append(p)
        assert f(bufs[0], n, ld, bufs[1], bufs[2]) == 0
        assert lib.irwls_dev_d2h(x.ctypes.data, bufs[2], x.nbytes) == 0
        assert lib.irwls_dev_d2h(L.ctypes.data, bufs[0], L.nbytes) == 0 and lib.irwls_dev_sync() == 0
        for p in bufs:
            lib.irwls_dev_free(p)
        r = (A.astype(np.longdouble) @ x - b).astype(float)
        assert np.linalg.norm(r) <= 8 * n * 2.0 ** -53 * np.linalg.norm(A, 2) * np.linalg.norm(x) + 1e-300
        out.append((x, np.tril(L[:, :n].T)))
    assert np.array_equal(out[0][1], out[1][1])
    assert np.array_equal(out[0][0], out[2][0])  # the ready list is left clean
