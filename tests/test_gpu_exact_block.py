"""IRWLSpar's kernel block from the tensor cores (irwls_exact_block) against extended
precision; the bound per value is that of the predictions (test_gpu_predict_tc.py)."""
import ctypes as C

import numpy as np
import pytest

from libirwls_gb300 import _abi, load

pytestmark = pytest.mark.gpu
VP, I = C.c_void_p, C.c_int
EPS = 2.0 ** -53


# rows and columns around the tiles, an odd leading dimension, several drains, rows past the first n
@pytest.mark.parametrize("n,d,m", [(3907, 20, 128), (1700, 100, 301), (641, 9, 800), (5000, 54, 129)])
def test_against_extended_precision(n, d, m):
    rng = np.random.default_rng(n)
    gamma, rows = 0.5, max(n, m) + 2
    X = rng.standard_normal((rows, d)) / np.sqrt(d) * 2.0 ** rng.integers(-3, 2, (rows, 1))
    X[rng.random(X.shape) < 0.3] = 0.0
    r, c = np.nonzero(X)
    hd = _abi.build_dataset(np.r_[0, np.cumsum(np.bincount(r, minlength=rows))], c + 1, X[r, c], np.ones(rows), False)
    q = hd.q[:rows].copy()
    lib, bufs = load(), []
    lib.irwls_dev_upload.argtypes = [VP, I, I, C.c_double, I, I, VP]
    lib.irwls_dev_malloc.argtypes = [C.POINTER(VP), C.c_size_t]
    lib.irwls_dev_h2d.argtypes = lib.irwls_dev_d2h.argtypes = [VP, VP, C.c_size_t]
    lib.irwls_dev_free.argtypes = lib.irwls_dev_release.argtypes = [VP]
    lib.irwls_exact_block.argtypes = [VP, I, VP, I, VP, C.c_longlong]
    S = (C.c_char * 256)()
    assert lib.irwls_dev_upload(C.byref(hd.struct), rows, 1, gamma, 0, 0, S) == 0

    def put(a):
        p = VP()
        assert lib.irwls_dev_malloc(C.byref(p), a.nbytes) == 0
        assert lib.irwls_dev_h2d(p, a.ctypes.data, a.nbytes) == 0 and lib.irwls_dev_sync() == 0
        bufs.append(p)
        return p

    idx = rng.choice(rows, m, replace=False).astype(np.int32)
    idx[:2] = rows - 2, rows - 1
    ldo = m + 3
    out = np.full((n, ldo), 7.0)
    di, do = put(idx), put(out)
    assert lib.irwls_exact_block(S, n, di, m, do, ldo) == 0
    assert lib.irwls_dev_d2h(out.ctypes.data, do, out.nbytes) == 0 and lib.irwls_dev_sync() == 0
    assert lib.irwls_tc_status() == 0
    for p in bufs:
        lib.irwls_dev_free(p)
    lib.irwls_dev_release(S)
    assert np.all(out[:, m:] == 7.0)
    pick = np.unique(np.r_[0, n - 1, rng.integers(0, n, 60)])
    L = np.longdouble
    k = np.exp(-L(gamma) * (q[pick, None].astype(L) + q[None, idx] - 2 * (X[pick].astype(L) @ X[idx].astype(L).T)))
    dot = d * 2.1 ** 2 * np.sqrt(q[pick, None]) * np.sqrt(q[None, idx]) * (2 * 2.0 ** -56 + 2.0 ** -61)
    top = 1.45 * gamma * 4 * q.max()
    rel = 2 * gamma * dot + 4 * max(2.0 ** -56, 2.0 ** -57 * top) + EPS
    assert np.all(np.abs(out[pick, :m] - k) <= k * rel)
