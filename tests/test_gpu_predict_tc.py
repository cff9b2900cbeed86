"""RBF predictions on the tensor cores (batches of at least 500000 kernel values)
against extended-precision sums, and the inputs that stay on the ordered path.

The bound, from the arithmetic: a feature is within 2^-56 of its row's scale
sigma (at most 2.1 times the row's norm), so a product's term moves by at most
2 x 2^-56 sigma_i sigma_j, and 2^-61 for the dropped digit levels; the
exponent's fixed point has 4 roundings of 2^-56 or 2^-57 of its largest term; a
kernel value and its product with the weight round twice, the sum nsv + 64
times."""
import ctypes as C

import numpy as np
import pytest

from libirwls_gb300 import _abi, load

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def _set(M, q=None):
    """The non-zero entries of M as a dataset (one index twice where q says so)."""
    n, d = M.shape
    r, c = np.nonzero(M)
    f = np.zeros(len(r) + n, dtype=_abi.SAMPLE_DTYPE)
    cnt = np.bincount(r, minlength=n)
    start = np.concatenate([[0], np.cumsum(cnt + 1)])
    pos = np.arange(len(r)) + r
    f["index"][pos], f["value"][pos] = c + 1, M[r, c]
    f["index"][start[1:] - 1] = -1
    q = np.einsum("ij,ij->i", M, M) if q is None else q
    return _abi.HostDataset(f, start[:-1], np.ones(n), q, n, 1, d)


def _model(S, w, gamma, bias):
    lib = load()
    beta = np.concatenate([w, [bias]])
    return lib.calculateFULLModel(_abi.make_properties(gamma=gamma), S.struct,
                                  beta.ctypes.data_as(C.POINTER(C.c_double)))


def _soft(T, mdl, n, soft=True):
    lib = load()
    f = lib.softTest if soft else lib.test
    return np.ctypeslib.as_array(f(T.struct, mdl, _abi.make_predict_properties()), shape=(n,)).copy()


def _data(kind, n, d, seed):
    rng = np.random.default_rng(seed)
    if kind == "onehot":
        return (rng.random((n, d)) < 0.2).astype(float)
    M = rng.standard_normal((n, d)) / np.sqrt(d)
    if kind == "scales":
        M *= 2.0 ** rng.integers(-8, 3, (n, 1))
        M[::5] = 0.0
    return M


# rows and vectors around the 128 x 64 tiles, features around the 16- and 96-feature blocks,
# exponents below and above 32 (the two fixed points)
@pytest.mark.parametrize("kind,n,d,nsv,gamma", [("dense", 16000, 1, 63, 0.4), ("scales", 7937, 16, 127, 0.4),
                                                ("dense", 1000, 17, 1001, 30.0),
                                                ("onehot", 129, 54, 7900, 0.1), ("dense", 127, 96, 8000, 0.4),
                                                ("scales", 4001, 97, 257, 2.0), ("dense", 1500, 300, 700, 0.4)])
def test_against_extended_precision(kind, n, d, nsv, gamma):
    rng = np.random.default_rng(d)
    bias = 0.25
    A, B, w = _data(kind, n, d, 1), _data(kind, nsv, d, 2), rng.standard_normal(nsv)
    T, S = _set(A), _set(B)
    mdl = _model(S, w, gamma, bias)
    pick = np.unique(np.concatenate([[0, n - 1], rng.integers(0, n, 50)]))
    L = np.longdouble
    D = T.q[pick, None].astype(L) + S.q[None, :] - 2 * (A[pick].astype(L) @ B.astype(L).T)
    k = np.exp(-L(gamma) * D)
    ref = k @ w.astype(L) + L(bias)
    sa, sb = 2.1 * np.sqrt(T.q[pick, None]), 2.1 * np.sqrt(S.q[None, :])
    dot = d * sa * sb * (2 * 2.0 ** -56 + 2.0 ** -61)
    top = 1.45 * gamma * (T.q.max() + S.q.max() + 2 * np.sqrt(T.q.max() * S.q.max()))
    rel = 2 * gamma * dot + 4 * max(2.0 ** -56, 2.0 ** -57 * top) + 2 * EPS
    tol = np.sum(np.abs(w) * k * rel, 1) + (nsv + 64) * EPS * (np.sum(np.abs(w) * k, 1) + bias)
    got = _soft(T, mdl, n)
    assert np.all(np.abs(got[pick] - ref) <= tol)
    # the ordered path on a few of the rows, and the labels
    few = _soft(_set(A[pick]), mdl, len(pick))
    assert np.all(np.abs(got[pick] - few) <= 2 * tol + 64 * d * EPS * top * np.sum(np.abs(w) * k, 1))
    assert np.array_equal(_soft(T, mdl, n, soft=False), np.where(got >= 0, 1.0, -1.0))


@pytest.mark.parametrize("what", ["weight", "scale", "gamma", "twice"])
def test_inputs_for_the_ordered_path(what):
    n, d, nsv = 9000, 9, 120
    A, B = _data("dense", n, d, 3), _data("dense", nsv, d, 4)
    w = np.random.default_rng(5).standard_normal(nsv)
    gamma = 0.3
    if what == "weight":
        w[7] = np.inf
    if what == "scale":
        A[11] *= 1e160
    if what == "gamma":
        gamma = 1e9
    S = _set(B)
    if what == "twice":
        S.features["index"][S.features["index"] == 5] = 4
    mdl = _model(S, w, gamma, 0.1)
    got = _soft(_set(A), mdl, n)
    parts = [_soft(_set(A[i:i + 3000]), mdl, min(3000, n - i)) for i in range(0, n, 3000)]
    assert np.array_equal(got, np.concatenate(parts), equal_nan=True)
