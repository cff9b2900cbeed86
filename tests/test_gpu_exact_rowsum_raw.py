"""Single kernel values of raw rows (dense sets in full training) from irwls_exact_rowsum,
a common offset making the rows' norms large against their differences.

A value's error: 2^-56 sigma per feature of either row, at most 2 c |d|_1 2^-55 sigma in the
exponent; the dropped digit levels, at most 1.25 units 2^-62 c sigma sigma' of T per feature in
each of the three products and two units more per 96 features; 4 units of y; 2 roundings."""
import ctypes as C

import numpy as np
import pytest

from libirwls_gb300 import _abi, load

pytestmark = pytest.mark.gpu
VP, I = C.c_void_p, C.c_int
N, NB = 2000, 300


# width, the exponent of twice a row's norm (about; the largest is up to 1.7 times that), the spread of the rows; whether they are for this path
@pytest.mark.parametrize("d,top,spread,taken", [(20, 15, 1.0, True), (40, 30, 0.2, True), (100, 12, 0.2, True),
                                                (97, 4, 1.0, True), (100, 17, 0.2, False), (4, 12, 0.2, True), (4, 45, 0.2, False),
                                                (20, 45, 0.2, True), (20, 90, 0.2, False), (200, 120, 0.2, False),
                                                (784, 62, 0.2, False), (784, 120, 1.0, False), (2000, 16, 0.2, False)])
def test_values(d, top, spread, taken):
    rng = np.random.default_rng(d)
    gamma, L = 1.0 / d, np.longdouble
    X = rng.standard_normal((N, d)) * spread + np.sqrt(max(0.0, top / 5.9 - spread ** 2))
    X[-NB:] = X[:NB] + 0.01 * rng.standard_normal((NB, d))  # rows near the vectors, beside the vectors themselves
    f = np.zeros(N * (d + 1), dtype=_abi.SAMPLE_DTYPE)
    f["index"], f["value"] = np.tile(np.r_[np.arange(d), -1], N), np.c_[X, np.zeros(N)].ravel()
    hd = _abi.HostDataset(f, np.arange(N) * (d + 1), np.ones(N), np.einsum("ij,ij->i", X, X), N, 0, d)
    lib, bufs = load(), []
    lib.irwls_dev_upload.argtypes = [VP, I, I, C.c_double, I, I, VP]
    lib.irwls_dev_malloc.argtypes = [C.POINTER(VP), C.c_size_t]
    lib.irwls_dev_h2d.argtypes = lib.irwls_dev_d2h.argtypes = [VP, VP, C.c_size_t]
    lib.irwls_dev_free.argtypes = lib.irwls_dev_release.argtypes = lib.irwls_exact_rows_free.argtypes = [VP]
    lib.irwls_exact_rows_create.restype, lib.irwls_exact_rows_create.argtypes = VP, [VP, I, I]
    lib.irwls_exact_rowsum.argtypes = [VP, VP, I, VP, VP, I, VP, VP, I, VP, VP, VP]
    S = (C.c_char * 256)()
    assert lib.irwls_dev_upload(C.byref(hd.struct), N, 1, gamma, 0, 0, S) == 0

    def put(a):
        p = VP()
        assert lib.irwls_dev_malloc(C.byref(p), a.nbytes) == 0
        assert lib.irwls_dev_h2d(p, a.ctypes.data, a.nbytes) == 0 and lib.irwls_dev_sync() == 0
        bufs.append(p)
        return p

    E = lib.irwls_exact_rows_create(S, N, NB)
    out = np.zeros(N)
    ib, nb, do = put(np.arange(NB, dtype=np.int32)), put(np.array([NB], np.int32)), put(out)
    c = 1.4427 * gamma
    norm = np.sqrt((X * X).sum(1))
    for j in (3, 77, 200) if E else ():
        w = np.zeros(NB)
        w[j] = 1.0
        assert lib.irwls_exact_rowsum(E, None, N, ib, nb, NB, put(w), None, 1, None, None, do) == 0
        assert lib.irwls_dev_d2h(out.ctypes.data, do, out.nbytes) == 0 and lib.irwls_dev_sync() == 0
        D = X.astype(L) - X[j].astype(L)
        k = np.exp(-L(gamma) * (D * D).sum(1))
        sig = 2.1 * np.maximum(norm, norm[j])
        y = (2 * c * np.abs(D).sum(1) * 2.0 ** -55 * sig + c * sig * sig * 2.0 ** -62 * (4 * 1.25 * d + 2 * (1 + d / 96))
             + 4 * 2.0 ** -53)
        err = (out - k).astype(float)
        assert np.all(np.abs(err) <= (0.7 * y + 2 * 2.0 ** -53) * k.astype(float))
    lib.irwls_exact_rows_free(E)
    for p in bufs:
        lib.irwls_dev_free(p)
    lib.irwls_dev_release(S)
    assert bool(E) == taken
