"""The FP64 Gram of small budgets (irwls_par_gram_fp64, fewer than 128 columns)
against extended-precision products: a chunk's multiply-adds round once each, the
P chunks' sums and KC add P + 1 roundings, and each product of a weight and a
kernel value rounds twice (both factors of a term)."""
import ctypes as C

import numpy as np
import pytest

from libirwls_gb300 import load

pytestmark = pytest.mark.gpu
VP = C.c_void_p


# one column, the edges of the 4 x 2 micro-tiles, of a warp's 32 and of the 16-row copies; chunks
# without a row; the largest size
@pytest.mark.parametrize("l,m,nact,P", [(40, 1, 17, 1), (50, 2, 33, 3), (70, 4, 64, 2), (300, 22, 300, 4),
                                        (90, 31, 5, 8), (900, 64, 801, 5), (2000, 100, 1999, 64), (1500, 127, 1100, 7)])
def test_against_exact_products(l, m, nact, P):
    rng = np.random.default_rng(l + m)
    KSC, KC = rng.standard_normal((l, m)), rng.standard_normal((m, m))
    act = np.sort(rng.choice(l, nact, replace=False)).astype(np.int32)
    sd, day = rng.uniform(0.1, 30.0, nact), rng.standard_normal(nact)
    lib = load()
    assert lib.irwls_dev_init() == 0
    lib.irwls_dev_malloc.argtypes = [C.POINTER(VP), C.c_size_t]
    lib.irwls_dev_h2d.argtypes = lib.irwls_dev_d2h.argtypes = [VP, VP, C.c_size_t]
    lib.irwls_dev_free.argtypes = [VP]
    lib.irwls_par_gram_part_bytes.restype, lib.irwls_par_gram_part_bytes.argtypes = C.c_size_t, [C.c_int, C.c_int]
    lib.irwls_par_gram_fp64.argtypes = [VP, C.c_int, VP, C.c_int, VP, VP, VP, VP, C.c_int, VP, C.c_int]
    ld = m + 1
    bufs = []

    def put(a, n=None):
        p = VP()
        assert lib.irwls_dev_malloc(C.byref(p), max(a.nbytes if n is None else n, 16)) == 0
        bufs.append(p)
        if n is None:
            assert lib.irwls_dev_h2d(p, a.ctypes.data, a.nbytes) == 0
        return p

    try:
        dK, da, ds, dy, dC, d1 = [put(a) for a in (KSC, act, sd, day, KC, np.zeros((ld, ld)))]
        part = put(None, lib.irwls_par_gram_part_bytes(m, P))
        assert lib.irwls_par_gram_fp64(dK, m, da, nact, ds, dy, dC, d1, ld, part, P) == 0
        K1 = np.empty((ld, ld))
        lib.irwls_dev_d2h(K1.ctypes.data, d1, K1.nbytes)
        assert lib.irwls_dev_sync() == 0, lib.irwls_last_error_message()
    finally:
        for p in bufs:
            lib.irwls_dev_free(p)
    A = np.concatenate([sd[:, None] * KSC[act], day[:, None]], 1).astype(np.longdouble)
    ref, mag = A.T @ A[:, :m], np.abs(A).T @ np.abs(A[:, :m])
    ref[:m] += KC
    mag[:m] += np.abs(KC)
    r, c = np.indices((m + 1, m))
    err = np.abs(np.where(c <= r, K1.T[:, :m] - ref, 0.0))
    assert np.all(err <= (nact + P + 4) * 2.0 ** -53 * mag)
