"""The order in which a full training takes its memory: what it can do without comes last, so
that it never keeps from the training what that needs, and a refusal there is no error."""
import ctypes as C

import numpy as np
import pytest

import harness as H
from libirwls_gb300 import _abi, load, synth

pytestmark = pytest.mark.gpu
PD = C.POINTER(C.c_double)


# large enough for the row sums on the tensor cores (500000 values); the plain and the precision form
# (real-valued data: no exact-integer products there)
@pytest.mark.parametrize("mixed", [0, 1])
def test_refusals(mixed):
    lib, n, w = load(), 2000, 400
    lib.irwls_debug_fail_alloc.argtypes, lib.irwls_debug_fail_alloc.restype = [C.c_longlong], None
    X, y = synth.two_gaussians(n, 8, 1, shift=0.9)
    s = synth.from_dense(X, y, keep_zeros=True)
    hd = _abi.build_dataset(s.indptr, s.indices, s.values, s.y)
    props = _abi.make_properties(gamma=0.1, C_=1.0, working_set=w)
    h = lib.irwls_resident_upload(hd.struct, props, 0)
    assert h

    def train():
        beta = np.zeros(n + 1)
        H.LIBC.srand(0)
        rc = lib.irwls_resident_full(h, props, beta.ctypes.data_as(PD))
        return rc, lib.irwls_last_error(), beta

    lib.irwls_set_precision(mixed)
    try:
        rc, _, want = train()  # (the context's scratch memory is there from here on)
        assert rc == 0
        survived = []
        for k in range(1, 60):
            lib.irwls_debug_fail_alloc(k)
            rc, err, beta = train()
            lib.irwls_debug_fail_alloc(0)
            survived.append(rc == 0)
            if rc:
                assert err == -3
            else:
                assert err == 0
                assert H.rel_err(beta, want) <= (1e-4 if mixed else H.REL_TOL)
        # the training makes fewer than 60 allocations; once it can do without one, it can without all later ones
        first = survived.index(True)
        assert first > 20 and all(survived[first:])
    finally:
        lib.irwls_debug_fail_alloc(0)
        lib.irwls_set_precision(0)
        lib.irwls_resident_free(h)
