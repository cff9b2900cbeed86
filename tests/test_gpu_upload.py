"""The dataset upload: rows walked by several threads (sets above 250000 entries),
the dense copy made on the device, rows that name a feature twice or out of
order (the last entry stays), and the first bad row reported."""
import ctypes as C

import numpy as np
import pytest

from libirwls_gb300 import _abi, load

pytestmark = pytest.mark.gpu


def _set(rows):
    """HostDataset of (indices, values) rows as they are given, unlabeled."""
    lens = [len(i) for i, _ in rows]
    start = np.cumsum([0] + [n + 1 for n in lens])
    f = np.zeros(start[-1], dtype=_abi.SAMPLE_DTYPE)
    q = np.zeros(len(rows))
    for k, (ix, v) in enumerate(rows):
        f["index"][start[k]:start[k] + len(ix)] = ix
        f["value"][start[k]:start[k] + len(ix)] = v
        f["index"][start[k + 1] - 1] = -1
        q[k] = float(np.dot(v, v))
    top = max([max(i) for i, _ in rows if len(i)] + [0])
    return _abi.HostDataset(f, start[:-1], np.ones(len(rows)), q, len(rows), 1, int(top))


def _rows(n, d, seed):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(n):
        ix = np.sort(rng.choice(np.arange(1, d + 1), size=rng.integers(0, min(d, 30) + 1), replace=False))
        out.append((ix.tolist(), rng.standard_normal(len(ix)).tolist()))
    return out


@pytest.mark.parametrize("n,d,nsv", [(1, 3, 2), (70, 9, 64), (6000, 41, 130), (20000, 60, 33)])
def test_predictions_from_uploaded_rows(n, d, nsv):
    lib = load()
    rng = np.random.default_rng(n)
    test_rows, sv_rows = _rows(n, d, 1), _rows(nsv, d - 1, 2)
    for k in range(0, n, 7):  # a feature twice, and out of order
        ix, v = test_rows[k]
        test_rows[k] = (ix + [2, 1, 2], v + [0.5, -0.25, 1.5])
    t, s = _set(test_rows), _set(sv_rows)
    w = rng.standard_normal(nsv)
    props = _abi.make_properties(gamma=0.05)
    mdl = lib.calculateFULLModel(props, s.struct, np.concatenate([w, [0.3]]).ctypes.data_as(C.POINTER(C.c_double)))
    got = np.ctypeslib.as_array(lib.softTest(t.struct, mdl, _abi.make_predict_properties()), shape=(n,)).copy()
    T, S = np.zeros((n, d + 1)), np.zeros((nsv, d + 1))
    for M, rows in ((T, test_rows), (S, sv_rows)):
        for k, (ix, v) in enumerate(rows):
            for i, x in zip(ix, v):
                M[k, i] = x  # the last entry stays
    K = np.exp(-0.05 * (t.q[:, None] + s.q[None, :] - 2.0 * T @ S.T))
    ref = K @ w + 0.3
    # nsv terms, each within a few roundings of its size
    assert np.all(np.abs(got - ref) <= 64 * nsv * 2.0 ** -53 * (np.abs(K) @ np.abs(w) + 1.0))


def test_the_first_bad_row_is_reported():
    lib = load()
    rows = _rows(24000, 60, 3)
    for k in (8000, 4321, 8999):
        rows[k] = ([1], [float("nan")])
    d = _set(rows)
    p = _abi.make_properties(gamma=0.1, working_set=50)
    assert not lib.trainFULL(d.struct, p)
    assert lib.irwls_last_error() == -4 and b"row 4321" in lib.irwls_last_error_message()
