"""The plain form's Gram (irwls_par_gram, 7 exact base-256 digits per entry on
the tensor cores) against exact products.

The bound per row of the product, from the arithmetic: an entry's fixed point
is within 2^-56 sigma of it (2 x 2^-56 sigma_i sigma_j per product), and the
dropped digit levels u <= 4 weigh at most sum_u (u + 1) 128^2 256^u / 2^110
< 2^-61 sigma_i sigma_j; the partials of the split-K chunks and KC are added
in FP64 (at most P + 2 roundings of values below the sum of magnitudes)."""
import ctypes as C

import numpy as np
import pytest

from libirwls_gb300 import load

pytestmark = pytest.mark.gpu
VP = C.c_void_p


def _gram(KSC, act, sd, day, KC, P):
    lib = load()
    lib.irwls_dev_malloc.argtypes = [C.POINTER(VP), C.c_size_t]
    lib.irwls_dev_h2d.argtypes = lib.irwls_dev_d2h.argtypes = [VP, VP, C.c_size_t]
    lib.irwls_dev_free.argtypes = [VP]
    for f in (lib.irwls_par_gram_bytes, lib.irwls_par_gram_part_bytes):
        f.restype, f.argtypes = C.c_size_t, [C.c_int, C.c_int]
    lib.irwls_par_gram.argtypes = [VP, C.c_int, VP, C.c_int, VP, VP, VP, VP, C.c_int, VP, C.c_int, VP]
    l, m = KSC.shape
    ld = m + 1
    bufs = []

    def put(a, n=None):
        p = VP()
        assert lib.irwls_dev_malloc(C.byref(p), max(a.nbytes if n is None else n, 16)) == 0
        bufs.append(p)
        if n is None and a.nbytes:
            assert lib.irwls_dev_h2d(p, a.ctypes.data, a.nbytes) == 0
        return p

    try:
        host = [np.ascontiguousarray(a) for a in (KSC, act.astype(np.int32), sd, day, KC, np.zeros((ld, ld)))]
        dK, da, ds, dy, dC, d1 = [put(a) for a in host]
        part, ws = put(None, lib.irwls_par_gram_part_bytes(m, P)), put(None, lib.irwls_par_gram_bytes(l, m))
        assert lib.irwls_par_gram(dK, m, da, len(act), ds, dy, dC, d1, ld, part, P, ws) == 0
        K1 = np.empty((ld, ld))
        lib.irwls_dev_d2h(K1.ctypes.data, d1, K1.nbytes)
        assert lib.irwls_dev_sync() == 0, lib.irwls_last_error_message()
    finally:
        for p in bufs:
            lib.irwls_dev_free(p)
    r, c = np.indices((m + 1, m))
    return np.where(c <= r, K1.T[:, :m], 0.0)


# one column, the edges of the 128 x 64 tiles and of the 16- and 128-row blocks, one and several chunks
@pytest.mark.parametrize("l,m,nact,P", [(40, 1, 17, 1), (600, 63, 127, 1), (1100, 64, 513, 2), (1600, 127, 1536, 3),
                                        (1030, 128, 1030, 1), (3000, 200, 2500, 8)])
def test_against_exact_products(l, m, nact, P):
    rng = np.random.default_rng(l + m)
    KSC = np.exp(-rng.uniform(0.0, 30.0, (l, m)))
    act = np.sort(rng.choice(l, nact, replace=False))
    sd = 10.0 ** rng.uniform(-2, 2, nact)
    day = rng.standard_normal(nact) * sd
    KC = rng.uniform(0.0, 1.0, (m, m))
    got = _gram(KSC, act, sd, day, KC, P)
    A = np.concatenate([sd[:, None] * KSC[act], day[:, None]], axis=1)
    sig = 2.0 ** np.ceil(np.log2(np.abs(A).max(0)))
    # exact: every entry split into a 26-bit head and a tail, the products and sums in integers
    E = np.round(A / sig * 2.0 ** 60).astype(object)
    N = np.array([[int(v) for v in row] for row in E], dtype=object)
    cols = sorted({0, m // 2, m - 1})
    for j in cols:
        for i in sorted({j, m, min(m, j + 1)}):
            ref = sum(int(a) * int(b) for a, b in zip(N[:, i], N[:, j]))
            ref = float(ref / 2 ** 120) * sig[i] * sig[j] + (KC[i, j] if i < m else 0.0)
            mag = float(np.abs(A[:, i] * A[:, j]).sum()) + 1.0
            bound = nact * (2.0 ** -61 + 2.0 ** -55) * sig[i] * sig[j] + (P + 4) * 2.0 ** -53 * mag
            assert abs(got[i, j] - ref) <= bound, (i, j, got[i, j] - ref, bound)


def test_no_active_rows_and_zero_columns():
    rng = np.random.default_rng(3)
    KSC, KC = rng.random((100, 70)), rng.random((70, 70))
    KSC[:, 5] = 0.0
    low = np.tril(np.ones((71, 70)), 0) > 0
    got = _gram(KSC, np.zeros(0, np.int32), np.zeros(0), np.zeros(0), KC, 4)
    assert np.array_equal(got[:70][low[:70]], KC[low[:70]]) and not got[70].any()
    got = _gram(KSC, np.arange(100), np.ones(100), np.ones(100), KC, 2)
    assert got[5, 5] == KC[5, 5] and np.isfinite(got).all()
