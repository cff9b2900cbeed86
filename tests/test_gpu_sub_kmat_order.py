"""Full training on rows that name a feature twice or out of order: the dense copy keeps the
last entry and the list has both, so k(i, j) and k(j, i) differ, and the kept kernel matrix
must hold what the direct path (working sets above 4096 rows) forms. (The two entries differ
little in effect: with very different ones the systems contradict the error updates, the
iteration does not settle, and any rounding shows.)"""
import numpy as np
import pytest

import harness as H
from libirwls_gb300 import _abi, load, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,what", [(60, "twice"), (300, "none"), (300, "twice"), (300, "order"), (700, "twice")])
def test_kept_and_direct(n, what):
    X, y = synth.two_gaussians(n, 6, 3)
    rows = [[(k + 1, X[i, k]) for k in range(6)] for i in range(n)]
    for r in rows[::3]:
        if what == "twice":
            r.append(r[1])
            r[1] = (2, 0.01 * r[0][1])
        if what == "order":
            r.reverse()
    f = np.zeros(sum(len(r) + 1 for r in rows), dtype=_abi.SAMPLE_DTYPE)
    f["index"] = [i for r in rows for i, _ in r + [(-1, 0.0)]]
    f["value"] = [v for r in rows for _, v in r + [(-1, 0.0)]]
    start = np.cumsum([0] + [len(r) + 1 for r in rows])[:-1]
    q = np.array([sum(v * v for _, v in r) for r in rows])
    hd = _abi.HostDataset(f, start, y.astype(float), q, n, 1, 6)
    lib, out = load(), []
    for w in (n + 100, 4200):  # (all rows fit both working sets)
        prop = _abi.make_properties(gamma=0.2, C_=3.0, working_set=w)
        lib.initMemory(1, w + 1)
        H.LIBC.srand(0)
        out.append(H.arr(lib.trainFULL(hd.struct, prop), n + 1))
    assert np.array_equal(out[0][:-1] != 0, out[1][:-1] != 0)
    assert H.rel_err(out[0], out[1]) <= H.REL_TOL
