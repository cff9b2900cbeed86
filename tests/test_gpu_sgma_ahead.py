"""The candidates' whitened kernel rows ahead of their steps (dev_sgma_ahead.cu):
w = L^-1 k_C(c) of every later candidate, eta, the bf16 images, Q's column and the
rows of the factor, for given choices, against extended-precision substitution.

The bound: kernel values are within (d + 8) eps (1 + 2 gamma |x|^2) of theirs, a sum
of s products within (s + 2) eps of its terms' magnitudes (at most 1: rows of L and
w have norms <= 1), an element divides by L_ss >= sqrt(jitter) and the error goes
through the substitution, whose inverse is bounded by the one computed here."""
import ctypes as C

import numpy as np
import pytest

from libirwls_gb300 import _abi, load

pytestmark = pytest.mark.gpu
VP = C.c_void_p
EPS = 2.0 ** -53


def _join(img, kbn, rows, piece):
    """(rows x 32 kbn) values of the blocked pieces."""
    b = img.reshape(-1, kbn, 3, piece // 256, 4, 8, 8).astype(np.uint32) << 16
    v = b.view(np.float32).astype(np.float64).sum(2)  # tile, block, r >> 3, c >> 3, r & 7, c & 7
    return v.transpose(0, 2, 4, 1, 3, 5).reshape(-1, 32 * kbn)[:rows]


# no later candidates, one step of them, the eight-warp split of the sums, several CTAs; wide rows
@pytest.mark.parametrize("l,d,m,raw,linear", [(40, 3, 2, 0, 0), (70, 5, 3, 0, 0), (300, 54, 20, 0, 0), (257, 9, 75, 1, 0),
                                              (129, 200, 34, 0, 0), (150, 6, 12, 0, 1)])
def test_substitution(l, d, m, raw, linear):
    rng = np.random.default_rng(l)
    gamma = 0.3
    X = rng.standard_normal((l + 2, d)) / np.sqrt(d) * 2
    if not raw:
        X[rng.random(X.shape) < 0.4] = 0.0
    f = np.zeros((l + 2) * (d + 1), dtype=_abi.SAMPLE_DTYPE)
    f["index"] = np.tile(np.r_[np.arange(0 if raw else 1, d + (0 if raw else 1)), -1], l + 2)
    f["value"] = np.c_[X, np.zeros(l + 2)].ravel()
    q = np.einsum("ij,ij->i", X, X)
    hd = _abi.HostDataset(f, np.arange(l + 2) * (d + 1), np.ones(l + 2), q, l + 2, 0 if raw else 1, d)
    lib, bufs = load(), []
    lib.irwls_dev_upload.argtypes = [VP, C.c_int, C.c_int, C.c_double, C.c_int, C.c_int, VP]
    lib.irwls_dev_malloc.argtypes = [C.POINTER(VP), C.c_size_t]
    lib.irwls_dev_h2d.argtypes = lib.irwls_dev_d2h.argtypes = [VP, VP, C.c_size_t]
    lib.irwls_dev_free.argtypes = lib.irwls_dev_release.argtypes = [VP]
    I, D = C.c_int, C.c_double
    lib.irwls_sgma_ahead_bytes.restype, lib.irwls_sgma_ahead_bytes.argtypes = C.c_size_t, [I, I]
    lib.irwls_sgma_ahead_init.argtypes = [VP, VP, I, I, VP]
    lib.irwls_sgma_factor.argtypes = [VP, I, VP, VP, VP, I, VP, I]
    lib.irwls_sgma_ahead_step.argtypes = [VP, I, VP, VP, VP, I, I, I, VP, VP, VP, VP, VP, VP, VP]
    S = (C.c_char * 256)()
    assert lib.irwls_dev_upload(C.byref(hd.struct), l + 2, 0 if linear else 1, gamma, 0, 0, S) == 0

    def put(a):
        p = VP()
        assert lib.irwls_dev_malloc(C.byref(p), max(a.nbytes, 16)) == 0
        assert lib.irwls_dev_h2d(p, a.ctypes.data, a.nbytes) == 0 and lib.irwls_dev_sync() == 0
        bufs.append(p)
        return p

    def get(p, a):
        assert lib.irwls_dev_d2h(a.ctypes.data, p, a.nbytes) == 0 and lib.irwls_dev_sync() == 0
        return a

    ldq, nc = 128 * ((m + 127) // 128), 64 * m
    cand = rng.integers(0, l, nc).astype(np.int32)
    slot = rng.integers(0, 64, m).astype(np.int32)
    cent = cand[64 * np.arange(m) + slot]
    cent[:2] = l, l + 1
    resid = rng.standard_normal((m, 64, l)).astype(np.float32)
    ws = put(np.zeros(lib.irwls_sgma_ahead_bytes(m, ldq), np.uint8))
    tiles = (l + 127) // 128
    dc, dt, db, dL = put(cand), put(cent), [put(slot[s:s + 1]) for s in range(m)], put(np.zeros((m, m)))
    dQ, deta, dr = put(np.zeros(tiles * 128 * ldq * 3, np.uint16)), put(np.zeros(64)), [put(r) for r in resid]
    assert lib.irwls_sgma_ahead_init(S, dc, m, ldq, ws) == 0
    etas = []
    for s in range(m):
        if s < 2:
            assert lib.irwls_sgma_factor(S, s, dt, db[s], None, m, dL, m) == 0
        assert lib.irwls_sgma_ahead_step(S, l, dc, dt, None if s < 2 else db[s], s, m, ldq, dL, ws, dQ, None, dr[s],
                                         deta, None) == 0
        etas.append(get(deta, np.zeros(64)))
    W, L = get(ws, np.zeros((m, nc))), get(dL, np.zeros((m, m)))
    img = get(VP(ws.value + nc * (m + 2) * 8), np.zeros(m * 64 * ldq * 3, np.uint16)).reshape(m, -1)
    Q = _join(get(dQ, np.zeros(tiles * 128 * ldq * 3, np.uint16)), ldq // 32, l, 128 * 32)
    for p in bufs:
        lib.irwls_dev_free(p)
    lib.irwls_dev_release(S)

    T = np.longdouble

    def kern(a, b):
        G = X[a].astype(T) @ X[b].astype(T).T
        return G if linear else np.exp(-T(gamma) * (q[a, None].astype(T) + q[None, b] - 2 * G))

    K, B = kern(cent, cand), kern(cent, cent)
    ref, R = np.zeros((m, nc), T), np.zeros((m, m), T)
    for s in range(m):
        R[s, :s] = ref[:s, 64 * s + slot[s]] if s >= 2 else (B[1, :1] / R[0, 0] if s else 0)
        R[s, s] = np.sqrt(B[s, s] + T(1e-6 if s == 0 else 1e-5) - (R[s, :s] ** 2).sum())
        ref[s] = (K[s] - R[s, :s] @ ref[:s]) / R[s, s]
    inv = np.abs(np.linalg.inv(R.astype(float))).sum(1).max()
    top = max(1.0, float(np.abs(B).max()))
    tol = inv * inv * EPS * ((d + 8) * (1 + 4 * gamma * q.max()) + m + 2) * top
    later = 64 * np.maximum(2, np.arange(m) + 1)
    for s in range(m):
        assert np.all(np.abs(W[s, later[s]:] - ref[s, later[s]:]) <= tol)
        if 2 <= s:
            assert np.all(np.abs(L[s, :s + 1] - R[s, :s + 1]) <= tol)
            want = (-resid[s, slot[s]] * np.float32(1.0 / L[s, s])).astype(np.float64)
            assert np.allclose(Q[:, s], want, rtol=2.0 ** -22, atol=0)
            w = W[:s, 64 * s:64 * s + 64].astype(np.float32)
            assert np.array_equal(_join(img[s], ldq // 32, 64, 64 * 32)[:, :s], w.T)
            assert np.all(np.abs(etas[s - 1] - (1 - (W[:s, 64 * s:64 * s + 64] ** 2).sum(0))) <= (s + 2) * EPS * 4 * top)
