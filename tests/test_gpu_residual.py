"""The error and weight update of IRWLSpar (irwls_par_residual) against
extended-precision sums: m multiply-adds and five additions round once each, the
weight C / (y e) three times more."""
import ctypes as C

import numpy as np
import pytest

from libirwls_gb300 import load

pytestmark = pytest.mark.gpu
VP = C.c_void_p


# the edges of a warp's 8 rows and 32 columns, one and several passes of the grid's warps
@pytest.mark.parametrize("l,m", [(1, 1), (7, 31), (8, 32), (9, 33), (63, 100), (1001, 300), (78001, 5)])
def test_errors_and_weights(l, m):
    rng = np.random.default_rng(l)
    K, beta, y = rng.standard_normal((l, m)), rng.standard_normal(m), np.where(rng.random(l) < 0.5, -1.0, 1.0)
    cost, top = 3.0, 1e4
    lib = load()
    assert lib.irwls_dev_init() == 0
    lib.irwls_dev_malloc.argtypes = [C.POINTER(VP), C.c_size_t]
    lib.irwls_dev_h2d.argtypes = lib.irwls_dev_d2h.argtypes = [VP, VP, C.c_size_t]
    lib.irwls_dev_free.argtypes = [VP]
    lib.irwls_par_residual.argtypes = [VP, C.c_int, C.c_int, VP, VP, C.c_double, C.c_double, VP, VP]
    bufs = []
    for a in (K, beta, y, np.zeros(l), np.zeros(l)):
        p = VP()
        assert lib.irwls_dev_malloc(C.byref(p), max(a.nbytes, 16)) == 0 and lib.irwls_dev_h2d(p, a.ctypes.data, a.nbytes) == 0
        bufs.append(p)
    dK, db, dy, de, da = bufs
    e, a = np.empty(l), np.empty(l)
    assert lib.irwls_par_residual(dK, l, m, db, dy, cost, top, de, da) == 0
    assert lib.irwls_dev_d2h(e.ctypes.data, de, e.nbytes) == 0 and lib.irwls_dev_d2h(a.ctypes.data, da, a.nbytes) == 0
    assert lib.irwls_dev_sync() == 0
    for p in bufs:
        lib.irwls_dev_free(p)
    L = np.longdouble
    ref = y - K.astype(L) @ beta.astype(L)
    assert np.all(np.abs(e - ref) <= (m + 7) * 2.0 ** -53 * (1 + np.abs(K) @ np.abs(beta)))
    with np.errstate(divide="ignore"):
        want = np.where(e * y < 0, 0.0, np.minimum(cost / (y * e), top))
    assert np.all(np.abs(a - want) <= 4 * 2.0 ** -53 * want)
