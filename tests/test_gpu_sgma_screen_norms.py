"""The screened selection on rows whose norms are large against 1 / gamma, where FP32 kernel
values are off by far more than in centred data: the centroids are those of the FP64 scores,
which verbose = 1 takes in every step."""
import numpy as np
import pytest

import harness as H
from libirwls_gb300 import _abi, load, synth

pytestmark = pytest.mark.gpu


def _sgma(hd, m, gamma, verbose):
    p = _abi.make_properties(gamma=gamma, C_=10.0, size=m, algorithm=1, verbose=verbose)
    load().initMemory(1, m)
    H.LIBC.srand(5)
    return H.arr(load().SGMA(hd.struct, p), m, np.int32)


# gamma |x|^2 from 10 to 10^5, kernel values of order one; raw rows and norms
@pytest.mark.parametrize("off", [5.0, 30.0, 500.0])
@pytest.mark.parametrize("zeros", [False, True])
def test_common_offset(off, zeros):
    X, y = synth.two_gaussians(1500, 20, 3)
    s = synth.from_dense(X + off, y, keep_zeros=zeros)
    hd = _abi.build_dataset(s.indptr, s.indices, s.values, s.y)
    assert np.array_equal(_sgma(hd, 50, 0.02, 0), _sgma(hd, 50, 0.02, 1))


@pytest.mark.parametrize("off", [64.0, 512.0])
def test_rare_rows_that_fp32_does_not_hold(off):
    """Integer rows in pairs about integer class means, which FP32 holds exactly, and a few that it rounds."""
    rng = np.random.default_rng(9)
    rows, y = [], []
    for c in (0, 1):
        D = rng.integers(-1, 2, (500, 20)).astype(float)
        D[:3] += rng.random((3, 20)) - 0.5
        rows += [off + c + D, off + c - D]
        y.append(np.full(1000, 1.0 - 2 * c))
    p = rng.permutation(2000)
    s = synth.from_dense(np.concatenate(rows)[p], np.concatenate(y)[p], keep_zeros=False)
    hd = _abi.build_dataset(s.indptr, s.indices, s.values, s.y)
    assert np.array_equal(_sgma(hd, 20, 0.1, 0), _sgma(hd, 20, 0.1, 1))
