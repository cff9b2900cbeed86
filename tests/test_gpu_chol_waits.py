"""The cluster sweep's waits running out (irwls_debug_sweep_wait): the solve ends, the
callers are told, and the next one is as if nothing had been. With no polls at all every
wait of every thread runs out; nothing is skipped but the waiting."""
import ctypes as C

import numpy as np
import pytest

import harness as H
from libirwls_gb300 import _abi, load

pytestmark = pytest.mark.gpu
PD = C.POINTER(C.c_double)


@pytest.fixture
def lib():
    lib = load()
    assert lib.irwls_gpu_available(), lib.irwls_last_error_message()
    lib.irwls_debug_sweep_wait.argtypes = [C.c_longlong]
    lib.irwls_debug_sweep_wait.restype = None
    yield lib
    lib.irwls_debug_sweep_wait(-1)


def _system(n):
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n)) / np.sqrt(n)
    return G @ G.T + np.eye(n), rng.standard_normal(n)


def _solve(lib, A, b):
    n = len(b)
    M, x = np.asfortranarray(A).ravel(order="F").copy(), np.full(n, 7.0)
    lib.ParallelLinearSystem(M.ctypes.data_as(PD), n, n, 0, 0, b.ctypes.data_as(PD), n, 1, 0, 0, n, 1,
                             x.ctypes.data_as(PD), n, 1, 0, 0, 1)
    return x


# two blocks (one CTA), two CTAs, eight with the last block partial, the largest order
@pytest.mark.parametrize("n", [64, 65, 501, 2048])
def test_solves(lib, n):
    torch = pytest.importorskip("torch")
    A, b = _system(n)
    solve = lib.irwls_chol_solve_noalloc
    solve.restype, solve.argtypes = C.c_int, [C.c_void_p, C.c_int, C.c_int] + [C.c_void_p] * 4
    right = _solve(lib, A, b)
    assert lib.irwls_last_error() == 0

    def noalloc():
        M = np.zeros((n, n + 1))
        M[:, :n] = A
        d = [torch.tensor(v, device="cuda") for v in (M, b, np.zeros(n))]
        info = torch.full((1,), 5, dtype=torch.int32, device="cuda")
        assert solve(d[0].data_ptr(), n, n + 1, d[1].data_ptr(), d[2].data_ptr(), info.data_ptr(),
                     torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        return int(info.item()), d[2].cpu().numpy()

    lib.irwls_debug_sweep_wait(0)
    assert np.array_equal(_solve(lib, A, b), np.full(n, 7.0)) and lib.irwls_last_error() == -13
    assert noalloc()[0] == -1
    lib.irwls_debug_sweep_wait(-1)
    info, x = noalloc()
    assert info == 0 and np.array_equal(x, right)
    assert np.array_equal(_solve(lib, A, b), right) and lib.irwls_last_error() == 0


def test_trainings(lib):
    g, gb = H.golden("full_sparse"), H.golden("budget_random")
    p, pb = H.params(g), H.params(gb)
    hd, hb = H.datasets(g)[0], H.datasets(gb)[0]
    lib.irwls_debug_sweep_wait(0)
    prop = _abi.make_properties(gamma=p["gamma"], C_=p["C"], kernel=p["kernel"], working_set=p["w"])
    lib.initMemory(1, p["w"] + 1)
    H.LIBC.srand(0)
    assert not lib.trainFULL(hd.struct, prop) and lib.irwls_last_error() == -13
    prop = _abi.make_properties(gamma=pb["gamma"], C_=pb["C"], kernel=pb["kernel"], size=pb["size"], algorithm=0)
    H.LIBC.srand(1)
    c = lib.randomCentroids(hb.struct, prop)
    assert not lib.IRWLSpar(hb.struct, c, prop) and lib.irwls_last_error() == -13
    lib.irwls_debug_sweep_wait(-1)
    beta, _, _ = H.run_full(lib, hd, p)
    assert H.rel_err(beta, g["beta"]) <= H.REL_TOL
    cent, w, _, _, _ = H.run_budget(lib, hb, pb)
    assert np.array_equal(cent, gb["centroids"]) and H.rel_err(w, gb["weights"]) <= H.REL_TOL
