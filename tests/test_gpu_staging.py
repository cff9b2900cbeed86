"""What the library keeps of its upload buffers: bounded, and given back by freeMemory."""
import ctypes as C
import threading

import numpy as np
import pytest

import harness as H
from libirwls_gb300 import _abi, load, synth

pytestmark = pytest.mark.gpu


def test_given_back():
    lib = load()
    lib.irwls_staging_bytes.restype = C.c_longlong
    s = synth.mixed_onehot(40000, 1)
    hd = _abi.build_dataset(s.indptr, s.indices, s.values, s.y)
    props = _abi.make_properties(gamma=0.1, working_set=50)
    for _ in range(2):
        handles = [lib.irwls_resident_upload(hd.struct, props, 0) for _ in range(6)]
        assert all(handles)
        for h in handles:
            lib.irwls_resident_free(h)
        assert 0 < lib.irwls_staging_bytes() <= 4 * (64 << 20)
        lib.freeMemory(1)
        assert lib.irwls_staging_bytes() == 0


def test_given_back_while_others_upload():
    lib = load()
    lib.irwls_staging_bytes.restype = C.c_longlong
    s = synth.mixed_onehot(3000, 2)
    hd = _abi.build_dataset(s.indptr, s.indices, s.values, s.y)
    n = 8
    ds, pr = (_abi.SvmDataset * n)(*[hd.struct] * n), (_abi.Properties * n)(
        *[_abi.make_properties(gamma=0.1, C_=1.0, working_set=100)] * n)
    PD = C.POINTER(C.c_double)
    betas = (PD * n)()
    out = []
    t = threading.Thread(target=lambda: out.append(lib.irwls_full_train_batch(ds, pr, None, n, 4, betas)))
    t.start()
    while t.is_alive():
        lib.irwls_staging_bytes()
        t.join(0.002)
        lib.freeMemory(1)
    assert out == [0]
    b = [H.arr(betas[i], hd.l + 1) for i in range(n)]
    assert all(np.array_equal(x, b[0]) for x in b)
    lib.freeMemory(1)
    assert lib.irwls_staging_bytes() == 0
