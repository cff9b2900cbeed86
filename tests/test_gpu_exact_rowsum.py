"""Row sums within one set on the tensor cores (irwls_exact_rowsum, the error
updates of plain full training) against extended precision; the bound is that of
the predictions (test_gpu_predict_tc.py)."""
import ctypes as C

import numpy as np
import pytest

from libirwls_gb300 import _abi, load

pytestmark = pytest.mark.gpu
VP, I = C.c_void_p, C.c_int
EPS = 2.0 ** -53


# all rows and a list of them; list
# lengths around the tiles, empty, the largest; one and several drains; raw rows
@pytest.mark.parametrize("n,d,na,nb,most,raw", [(4001, 20, 0, 500, 500, 0), (1000, 54, 0, 127, 600, 0),
                                                (3000, 7, 190, 2811, 2900, 0), (2000, 100, 300, 65, 2000, 0),
                                                (1500, 97, 0, 0, 400, 0), (4001, 20, 0, 500, 500, 1),
                                                (800, 130, 700, 700, 720, 0), (900, 130, 800, 640, 700, 1),
                                                (800, 5, 0, 30, 100, 0)])
def test_against_extended_precision(n, d, na, nb, most, raw):
    rng = np.random.default_rng(n)
    gamma = 0.5
    X = rng.standard_normal((n, d)) / np.sqrt(d) * 2.0 ** rng.integers(-3, 2, (n, 1))
    X[rng.random(X.shape) < 0.3] = 0.0
    r, c = np.nonzero(X)
    if raw:
        f = np.zeros(n * (d + 1), dtype=_abi.SAMPLE_DTYPE)
        f["index"], f["value"] = np.tile(np.r_[np.arange(d), -1], n), np.c_[X, np.zeros(n)].ravel()
        hd = _abi.HostDataset(f, np.arange(n) * (d + 1), np.ones(n), np.einsum("ij,ij->i", X, X), n, 0, d)
    else:
        hd = _abi.build_dataset(np.r_[0, np.cumsum(np.bincount(r, minlength=n))], c + 1, X[r, c], np.ones(n), False)
    q = hd.q[:n].copy()
    lib, bufs = load(), []
    lib.irwls_dev_upload.argtypes = [VP, I, I, C.c_double, I, I, VP]
    lib.irwls_dev_malloc.argtypes = [C.POINTER(VP), C.c_size_t]
    lib.irwls_dev_h2d.argtypes = lib.irwls_dev_d2h.argtypes = [VP, VP, C.c_size_t]
    lib.irwls_dev_free.argtypes = lib.irwls_dev_release.argtypes = lib.irwls_exact_rows_free.argtypes = [VP]
    lib.irwls_exact_rows_create.restype, lib.irwls_exact_rows_create.argtypes = VP, [VP, I, I]
    lib.irwls_exact_rowsum.argtypes = [VP, VP, I, VP, VP, I, VP, VP, I, VP, VP, VP]
    S = (C.c_char * 256)()
    assert lib.irwls_dev_upload(C.byref(hd.struct), n, 1, gamma, 0, 0, S) == 0

    def put(a):
        p = VP()
        assert lib.irwls_dev_malloc(C.byref(p), max(a.nbytes, 16)) == 0
        assert lib.irwls_dev_h2d(p, a.ctypes.data, a.nbytes) == 0 and lib.irwls_dev_sync() == 0
        bufs.append(p)
        return p

    rows = np.sort(rng.choice(n, na, replace=False)) if na else np.arange(n)
    ib = np.full(most, 2 ** 30, np.int32)  # (entries past the count are not read)
    ib[:nb] = np.sort(rng.choice(n, nb, replace=False))
    cb, sa = np.full(most, np.nan), np.where(rng.random(n) < 0.5, -1.0, 1.0)
    cb[:nb] = rng.standard_normal(nb)
    init, tail = rng.standard_normal(len(rows)), 0.75
    E = lib.irwls_exact_rows_create(S, n, max(na, 1))
    assert E
    dia = put(rows.astype(np.int32)) if na else None
    dib, dnb, dcb, dsa, dini, dt = [put(a) for a in (ib, np.array([nb], np.int32), cb, sa, init, np.array([tail]))]
    out = np.zeros(len(rows))
    do = put(out)
    small = len(rows) * most < 500000
    if na:
        rc = lib.irwls_exact_rowsum(E, dia, na, dib, dnb, most, dcb, dsa, 1, None, None, do)
    else:
        rc = lib.irwls_exact_rowsum(E, None, n, dib, dnb, most, dcb, None, -1, dini, dt, do)
    assert rc == (1 if small else 0)
    assert lib.irwls_dev_d2h(out.ctypes.data, do, out.nbytes) == 0 and lib.irwls_dev_sync() == 0
    assert lib.irwls_tc_status() == 0
    lib.irwls_exact_rows_free(E)
    for p in bufs:
        lib.irwls_dev_free(p)
    lib.irwls_dev_release(S)
    if small:
        return
    L, B = np.longdouble, ib[:nb]
    pick = np.unique(np.r_[0, len(rows) - 1, rng.integers(0, len(rows), 40)])
    ra, w = rows[pick], np.abs(cb[:nb])
    if raw:  # the distances themselves, not the rounded norms
        q = (X.astype(L) ** 2).sum(1)
    k = np.exp(-L(gamma) * (q[ra, None].astype(L) + q[None, B] - 2 * (X[ra].astype(L) @ X[B].astype(L).T)))
    q = q.astype(float)
    s = k @ cb[:nb].astype(L)
    ref = s * sa[ra] if na else init[pick] - s - L(tail)
    dot = d * 2.1 ** 2 * np.sqrt(q[ra, None]) * np.sqrt(q[None, B]) * (2 * 2.0 ** -56 + 2.0 ** -61)
    top = 1.45 * gamma * 4 * q.max()
    rel = 2 * gamma * dot + 4 * max(2.0 ** -56, 2.0 ** -57 * top) + 2 * EPS
    tol = np.sum(w * k * rel, 1) + (nb + 64) * EPS * (np.sum(w * k, 1) + np.abs(init[pick]) + tail)
    assert np.all(np.abs(out[pick] - ref) <= tol)
