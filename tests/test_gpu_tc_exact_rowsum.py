"""Row sums and kernel blocks with exact-integer tensor-core dot products
(irwls_tc_exact_rowsum, irwls_tc_exact_block) against extended precision: both forms
of the exponent, fixed point and FP64."""
import ctypes as C

import numpy as np
import pytest

from libirwls_gb300 import _abi, load

pytestmark = pytest.mark.gpu
VP, I, LL = C.c_void_p, C.c_int, C.c_longlong
EPS = 2.0 ** -53


# list lengths around the item widths (32, 64, 128) and empty; one value of 1, small
# integers of both signs, images; exponents on both sides of the fixed point's
# range; a row whose norm is not its own (its tiles take FP64)
@pytest.mark.parametrize("n,d,na,nb,kind,gamma,odd", [(300, 54, 129, 33, "one", 0.5, False), (300, 54, 128, 16, "one", 0.5, False),
                                                      (300, 54, 1, 1, "int", 0.003, False), (9000, 40, 9000, 130, "int", 0.01, True),
                                                      (12000, 33, 12000, 257, "one", 2.0 ** -40, False),
                                                      (3000, 100, 3000, 250, "img", 0.04, False), (500, 784, 400, 95, "img", 0.01, True),
                                                      (500, 40, 200, 64, "int", 0.5, False), (300, 20, 200, 0, "one", 0.5, False)])
def test_against_extended_precision(n, d, na, nb, kind, gamma, odd):
    rng = np.random.default_rng(n + d)
    K = (rng.random((n, d)) < 0.25) * (1 if kind == "one" else rng.integers(-9, 10, (n, d)) if kind == "int"
                                       else rng.integers(0, 256, (n, d)))
    K[:, 0] = 1
    s = 255 if kind == "img" else 1
    X = K / float(s)
    r, c = np.nonzero(X)
    hd = _abi.build_dataset(np.r_[0, np.cumsum(np.bincount(r, minlength=n))], c + 1, X[r, c], np.ones(n), False)
    if odd:
        hd.q[5] = -0.25
    q = hd.q[:n].copy()
    lib, bufs = load(), []
    lib.irwls_dev_upload.argtypes = [VP, I, I, C.c_double, I, I, VP]
    lib.irwls_dev_malloc.argtypes = [C.POINTER(VP), C.c_size_t]
    lib.irwls_dev_h2d.argtypes = lib.irwls_dev_d2h.argtypes = [VP, VP, C.c_size_t]
    lib.irwls_dev_free.argtypes = lib.irwls_dev_release.argtypes = lib.irwls_tc_set_free.argtypes = [VP]
    lib.irwls_tc_set_create.restype, lib.irwls_tc_set_create.argtypes = VP, [VP, I, I]
    lib.irwls_tc_set_exact.argtypes = [VP]
    lib.irwls_tc_exact_rowsum.argtypes = [VP, VP, VP, I, VP, I, VP, I, VP, VP, VP, I, VP, VP, VP]
    lib.irwls_tc_exact_block.argtypes = [VP, VP, VP, I, VP, I, VP, VP, VP, LL, I]
    assert lib.irwls_dev_init() == 0
    S = (C.c_char * 256)()
    assert lib.irwls_dev_upload(C.byref(hd.struct), n, 1, gamma, 0, 0, S) == 0

    def put(a):
        p = VP()
        assert lib.irwls_dev_malloc(C.byref(p), max(a.nbytes, 16)) == 0
        assert lib.irwls_dev_h2d(p, a.ctypes.data, a.nbytes) == 0 and lib.irwls_dev_sync() == 0
        bufs.append(p)
        return p

    ia, ib = np.sort(rng.choice(n, na, replace=False)).astype(np.int32), rng.choice(n, nb, replace=False).astype(np.int32)
    cb, init, out, blk = rng.standard_normal(nb), rng.standard_normal(na), np.zeros(na), np.zeros((max(nb, 1), na))
    T = lib.irwls_tc_set_create(S, n, 300)
    assert T and lib.irwls_tc_set_exact(T) == 1
    dia, dib, dcb, dini, do, dblk = [put(a) for a in (ia, ib, cb, init, out, blk)]
    assert lib.irwls_tc_exact_rowsum(T, S, dia, na, dib, nb, None, nb, dcb, None, None, -1, dini, None, do) == 0
    assert lib.irwls_tc_exact_block(T, S, dia, na, dib, nb, None, None, dblk, na, 0) == 0
    assert lib.irwls_dev_d2h(out.ctypes.data, do, out.nbytes) == 0
    assert lib.irwls_dev_d2h(blk.ctypes.data, dblk, blk.nbytes) == 0 and lib.irwls_dev_sync() == 0
    assert lib.irwls_tc_status() == 0
    lib.irwls_tc_set_free(T)
    for p in bufs:
        lib.irwls_dev_free(p)
    lib.irwls_dev_release(S)
    L = np.longdouble
    pick = np.unique(np.r_[0, na - 1, np.flatnonzero(ia == 5), rng.integers(0, na, 60)])
    dot = (K[ia[pick]] @ K[ib].T).astype(L) / L(s * s)
    qa, qb = q[ia[pick], None].astype(L), q[None, ib].astype(L)
    k = np.exp(-L(gamma) * (qa + qb - 2 * dot))
    # 2^-y and its rounding: 2 EPS, the fixed point's terms: 3 units of 2^-56; the FP64
    # form: three roundings of the exponent's terms and the scaled product's two
    rel = 2 * EPS + 4 * 2.0 ** -56 + 5 * EPS * gamma * (np.abs(qa) + np.abs(qb) + 2 * np.abs(dot))
    if nb:
        # (values below the normal doubles have no relative bound: small they are)
        normal, got = k >= 2.0 ** -1022, blk.T[pick]
        assert np.all(np.abs(got - k)[normal] <= (k * rel)[normal]) and np.all(np.abs(got[~normal]) <= 2.0 ** -1022)
    w = np.abs(cb)
    tol = (w * k * rel).sum(1) + (nb + 64) * EPS * ((w * k).sum(1) + np.abs(init[pick]))
    assert np.all(np.abs(out[pick] - (init[pick] - k @ cb.astype(L))) <= tol)
