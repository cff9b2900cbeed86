"""Timed work of the library: full and budgeted SVM training, prediction and
dense solves, each through the entry points a program calls.

Data are seeded: two Gaussian classes written with every feature (the dense
kernel form), continuous plus one-hot features (the sparse form) and 8-bit
prototype images with 784 features, the three kinds of ``libirwls_gb300.synth``.
"""
import ctypes as C
import math

import numpy as np
import torch

from libirwls_gb300 import LIBIRWLS, _abi, check, load, synth

LIBC = C.CDLL(None)
LIBC.free.argtypes = [C.c_void_p]
PD = C.POINTER(C.c_double)
PI = C.POINTER(C.c_int)
VP = C.c_void_p

GAMMA = {"dense": 0.05, "onehot": 0.1, "image": 0.02}
WIDTH = {"onehot": 54, "image": 784}
STORED = {"onehot": 12, "image": 150}  # stored values of a row, about


def listed():
    return [
        # one small SPD system already on the GPU: a caller's own iteration around a tiny budget
        dict(name="solve_order_64", kind="solve", order=64),
        # the system of one IRWLS iteration at a budget of 1000 centroids
        dict(name="solve_order_1000", kind="solve", order=1000),
        # a small table of mixed features through the C API with host data
        dict(name="full_onehot_700x54", kind="full", data="onehot", rows=700, dim=54, set=100, cost=10.0,
             mixed=False, entry="host"),
        # the dense full-IRWLS workload of the benchmark (4000 x 20, working set 500), data resident
        dict(name="full_dense_4000x20", kind="full", data="dense", rows=4000, dim=20, set=500, cost=10.0,
             mixed=False, entry="resident"),
        # images in the precision form, working set 500, data resident
        dict(name="full_image_20000_mixed", kind="full", data="image", rows=20000, dim=784, set=500, cost=10.0,
             mixed=True, entry="resident"),
        # budgeted training with random centroids through the C API with host data
        dict(name="budget_random_50000_m300", kind="budget", data="onehot", rows=50000, dim=54, size=300, sgma=False,
             cost=100.0, mixed=False, entry="host"),
        # budgeted training with SGMA centroids, the plain form, data resident
        dict(name="budget_sgma_20000_m100", kind="budget", data="onehot", rows=20000, dim=54, size=100, sgma=True,
             cost=100.0, mixed=False, entry="resident"),
        # the same in the precision form on more rows with a larger budget
        dict(name="budget_sgma_60000_m400_mixed", kind="budget", data="onehot", rows=60000, dim=54, size=400,
             sgma=True, cost=100.0, mixed=True, entry="resident"),
        # a few rows through the Python module: an online caller
        dict(name="predict_module_64x400", kind="predict", data="dense", rows=64, dim=20, vectors=400, linear=False,
             mixed=False, soft=True, entry="module"),
        # a whole test set against a full SVM's support vectors, the model kept on the GPU
        dict(name="predict_onehot_20000x3000", kind="predict", data="onehot", rows=20000, dim=54, vectors=3000,
             linear=False, mixed=False, soft=True, entry="device"),
        # labels of a linear model, model and rows on the host
        dict(name="predict_linear_9000x1501", kind="predict", data="dense", rows=9000, dim=33, vectors=1501,
             linear=True, mixed=False, soft=False, entry="host"),
        # images in the precision form, through the C API with host data
        dict(name="predict_image_8000x2000_mixed", kind="predict", data="image", rows=8000, dim=784, vectors=2000,
             linear=False, mixed=True, soft=True, entry="host"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "full", "full", "budget", "budget", "budget", "predict", "predict"])
    if kind == "solve":
        return dict(kind=kind, order=_log(rng, 16, 1500))
    if kind == "full":
        data = rng.choice(["dense", "onehot", "image"])
        case = dict(kind=kind, data=data, rows=_log(rng, 300, 3000), dim=WIDTH.get(data) or _log(rng, 4, 40),
                    set=_log(rng, 60, 500), cost=rng.choice([1.0, 10.0]), mixed=False,
                    entry=rng.choice(["host", "resident"]))
        if data == "image":
            case.update(rows=_log(rng, 2000, 20000), mixed=True, entry="resident")
        return case
    if kind == "budget":
        mixed, sgma = rng.random() < 0.3, rng.random() < 0.5
        rows = _log(rng, 1500, 60000 if mixed else 20000 if sgma else 50000)
        size = min(_log(rng, 20, 400 if mixed else 100 if sgma else 300), rows // 10)
        return dict(kind=kind, data="onehot", rows=rows, dim=54, size=size, sgma=sgma,
                    cost=100.0, mixed=mixed, entry=rng.choice(["host", "resident"]))
    data = rng.choice(["dense", "onehot", "image"])
    mixed = rng.random() < (0.5 if data == "image" else 0.25)
    most = 8000 if data == "image" else 20000
    entry = rng.choice(["module", "host"] if mixed else ["module", "host", "device"])
    return dict(kind=kind, data=data, rows=_log(rng, 20, most), dim=WIDTH.get(data) or _log(rng, 4, 60),
                vectors=_log(rng, 20, 2000 if data == "image" else 3000), linear=not mixed and rng.random() < 0.25,
                mixed=mixed, soft=rng.random() < 0.7, entry=entry)


def _matrix(case, rows, seed):
    if case["data"] == "dense":
        return synth.two_gaussians(rows, case["dim"], seed)
    if case["data"] == "onehot":
        s = synth.mixed_onehot(rows, seed)
        return s.dense(), s.y
    return synth.proto_digits(rows, seed)


class _Data:
    """A dataset struct and whoever owns its arrays."""

    def __init__(self, X, y, dense, means):
        self.lib = load()
        if dense:
            s = synth.from_dense(X, y, keep_zeros=True)
            self.own = _abi.build_dataset(s.indptr, s.indices, s.values, s.y, with_means=means)
            self.struct = self.own.struct
        else:
            self.own = None
            X, y = np.ascontiguousarray(X), np.ascontiguousarray(y)
            f = self.lib.irwls_dataset_from_dense_with_means if means else self.lib.irwls_dataset_from_dense
            self.struct = f(X.ctypes.data_as(PD), y.ctypes.data_as(PD), X.shape[0], X.shape[1])

    def __del__(self):
        if self.own is None:
            self.lib.freeDataset(self.struct)


class _Resident:
    """A training set kept on the GPU."""

    def __init__(self, data, props, means):
        self.lib, self.data = load(), data
        self.handle = check(self.lib.irwls_resident_upload(data.struct, props, int(means)), "irwls_resident_upload")

    def __del__(self):
        self.lib.irwls_resident_free(self.handle)


class _DeviceModel:
    def __init__(self, resident, props, beta):
        self.lib = load()
        self.handle = check(self.lib.irwls_dmodel_full(resident.handle, props, beta.ctypes.data_as(PD)), "irwls_dmodel_full")

    def __del__(self):
        self.lib.irwls_dmodel_free(self.handle)


def _spd(case, seed):
    """Kernel matrix of random points with a regularised diagonal, and a right-hand side."""
    rng = np.random.default_rng([seed, case["order"]])
    P = torch.from_numpy(rng.standard_normal((case["order"], 6))).cuda()
    sq = (P * P).sum(1)
    A = torch.exp(-0.1 * (sq[:, None] + sq[None, :] - 2.0 * P @ P.T).clamp_min(0.0))
    d = torch.from_numpy(rng.uniform(0.05, 2.0, case["order"])).cuda()
    return A + torch.diag(d), torch.from_numpy(rng.standard_normal(case["order"])).cuda()


def _weights(y, cost, rng):
    """Dual weights as a training leaves them: many at the bound, the others spread below it, and a bias."""
    a = np.where(rng.random(len(y)) < 0.4, cost, cost * rng.random(len(y)))
    return np.ascontiguousarray(np.concatenate([a * y, [0.25]]))


def prepare(case, seed):
    lib, kind = load(), case["kind"]
    if kind == "solve":
        A, b = _spd(case, seed)
        n = case["order"]
        f = lib.irwls_chol_solve_noalloc
        f.restype, f.argtypes = C.c_int, [VP, C.c_int, C.c_int, VP, VP, VP, VP]
        return dict(case=case, solve=f, A=A, b=b, M=torch.zeros(n, n + 1, dtype=torch.float64, device="cuda"),
                    x=torch.zeros(n, dtype=torch.float64, device="cuda"),
                    info=torch.zeros(1, dtype=torch.int32, device="cuda"))
    state = dict(case=case, seed=seed % 100003 + 1)
    if kind in ("full", "budget"):
        X, y = _matrix(case, case["rows"], seed)
        props = _abi.make_properties(gamma=GAMMA[case["data"]], C_=case["cost"], working_set=case.get("set", 500),
                                     size=case.get("size", 10), algorithm=int(case.get("sgma", False)))
        state["props"] = props
        means = kind == "budget"
        state["data"] = _Data(X, y, case["data"] == "dense", means)
        if case["entry"] == "resident":
            state["resident"] = _Resident(state["data"], props, means)
        return state
    rng = np.random.default_rng([seed, 7])
    X, y = _matrix(case, case["rows"] + case["vectors"], seed)
    T, S = X[:case["rows"]], X[case["rows"]:]
    props = _abi.make_properties(gamma=GAMMA[case["data"]], C_=10.0, kernel=0 if case["linear"] else 1)
    beta = _weights(y[case["rows"]:], 10.0, rng)
    vectors = _Data(S, y[case["rows"]:], False, False)
    if case["entry"] == "device":
        state["model"] = _DeviceModel(_Resident(vectors, props, False), props, beta)
    else:
        state["model"] = LIBIRWLS.Classifier(lib.calculateFULLModel(props, vectors.struct, beta.ctypes.data_as(PD)))
    if case["entry"] == "module":
        state["X"] = T
    else:
        state["data"] = _Data(T, y[:case["rows"]], False, False)
    state["props"] = _abi.make_predict_properties(labels=0, soft=int(case["soft"]))
    return state


def _take(ptr, n, what):
    out = np.ctypeslib.as_array(check(ptr, what), shape=(n,)).copy()
    LIBC.free(C.cast(ptr, VP))
    return out


def _train_full(lib, s):
    case, props = s["case"], s["props"]
    LIBC.srand(s["seed"])
    if case["entry"] == "host":
        lib.initMemory(1, props.MaxSize + 1)
        return {"beta": _take(lib.trainFULL(s["data"].struct, props), case["rows"] + 1, "trainFULL")}
    beta = np.empty(case["rows"] + 1)
    check(lib.irwls_resident_full(s["resident"].handle, props, beta.ctypes.data_as(PD)) == 0, "irwls_resident_full")
    return {"beta": beta}


def _train_budgeted(lib, s):
    case, props = s["case"], s["props"]
    m = case["size"]
    LIBC.srand(s["seed"])
    if case["entry"] == "resident":
        cent, w = np.empty(m, dtype=np.int32), np.empty(m)
        check(lib.irwls_resident_budgeted(s["resident"].handle, props, cent.ctypes.data_as(PI),
                                          w.ctypes.data_as(PD)) == 0, "irwls_resident_budgeted")
        return {"centroids": cent, "weights": w}
    ds = s["data"].struct
    lib.initMemory(1, m)
    c = lib.SGMA(ds, props) if case["sgma"] else lib.randomCentroids(ds, props)
    w = check(lib.IRWLSpar(ds, check(c, "centroids"), props), "IRWLSpar")
    return {"centroids": _take(c, m, "centroids"), "weights": _take(w, m, "IRWLSpar")}


def _predict(lib, s):
    case, m = s["case"], s["model"]
    if case["entry"] == "module":
        return LIBIRWLS.predict(m, s["X"], Soft=int(case["soft"]), verbose=0)
    ds = s["data"].struct
    if case["entry"] == "device":
        f = lib.irwls_dmodel_predict(m.handle, ds, s["props"], int(case["soft"]))
    else:
        f = (lib.softTest if case["soft"] else lib.test)(ds, m.model, s["props"])
    return _take(f, case["rows"], "prediction")


def run(state):
    case, lib = state["case"], load()
    if case["kind"] == "solve":
        n = case["order"]
        state["M"][:, :n].copy_(state["A"])  # the solve leaves the factor in its matrix
        rc = state["solve"](state["M"].data_ptr(), n, n + 1, state["b"].data_ptr(), state["x"].data_ptr(),
                            state["info"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        check(rc == 0, "irwls_chol_solve_noalloc")
        return {"x": state["x"], "info": state["info"]}
    lib.irwls_set_precision(1 if case["mixed"] else 0)
    return {"full": _train_full, "budget": _train_budgeted, "predict": _predict}[case["kind"]](lib, state)


def work(case):
    """Bytes and operations of the task itself: inputs read once, outputs written once; kernel values, systems and sums formed once."""
    kind = case["kind"]
    if kind == "solve":
        n = case["order"]
        return {"bytes": 8.0 * (n * n + 2 * n), "flops": n ** 3 / 3.0 + 2.0 * n * n}
    stored = STORED.get(case["data"], case["dim"])
    rows = 12.0 * stored * case["rows"]
    if kind == "full":
        # about 20 passes of working-set systems and error updates
        n, w = case["rows"], min(case["set"], case["rows"])
        return {"bytes": rows + 16.0 * n, "flops": 20.0 * (5 * w ** 3 / 3.0 + 2.0 * stored * n * w)}
    if kind == "budget":
        # K_nm once, about 20 systems; with SGMA 64 scored candidates at every order below the budget
        n, m = case["rows"], case["size"]
        flops = 2.0 * stored * n * m + 20.0 * (float(n) * m * m + m ** 3 / 3.0)
        return {"bytes": rows + 16.0 * n, "flops": flops + (64.0 * n * m * m if case["sgma"] else 0.0)}
    n, v = case["rows"], case["vectors"]
    return {"bytes": rows + 12.0 * stored * v + 8.0 * (n + v), "flops": 2.0 * stored * n * v + 2.0 * n * v}


def _exact_budgeted(case, seed):
    """IRWLS on the K_nm of random centroids (src/budgeted-train.c:324-505), in 64 bits on the GPU."""
    X, y = _matrix(case, case["rows"], seed)
    n, m, cost = case["rows"], case["size"], case["cost"]
    LIBC.srand(seed % 100003 + 1)
    p = np.arange(n)
    for i in range(n - 1, -1, -1):
        j = LIBC.rand() % (i + 1)
        p[i], p[j] = p[j], p[i]
    cent = p[:m].astype(np.int32)
    X, y = torch.from_numpy(X).cuda(), torch.from_numpy(y).cuda()
    sq = (X * X).sum(1)
    ix = torch.from_numpy(cent.astype(np.int64)).cuda()
    K = torch.exp(-GAMMA[case["data"]] * (sq[:, None] + sq[ix][None, :] - 2.0 * X @ X[ix].T))
    KC = K[ix] + 1e-5 * torch.eye(m, dtype=torch.float64, device="cuda")
    M, iters, since, old, best, dw, nw = 1e4, 0, 0, 0.0, 1e9, 1e9, 1.0
    beta = torch.zeros(m, dtype=torch.float64, device="cuda")
    A, day, bb = K, y * M, beta
    while iters < 500 and dw / nw > 1e-6 and since < 5:
        L = torch.linalg.cholesky(KC + A.T @ A)
        new = torch.cholesky_solve((A.T @ day)[:, None], L)[:, 0]
        dw, nw = float(((new - beta) ** 2).sum()), float((new ** 2).sum())
        beta = new
        e = y - K @ beta
        D = torch.where(e * y < 0.0, torch.zeros_like(e), cost / (y * e)).clamp_max(M)
        on = D != 0.0
        r = torch.sqrt(D[on])
        A, day = r[:, None] * K[on], r * y[on]
        iters += 1
        if iters > 10 and dw / nw > 100 * old:
            M /= 10.0
        old = dw / nw
        if dw / nw < best:
            best, since, bb = dw / nw, 0, new
        else:
            since += 1
    return {"centroids": cent, "weights": bb}


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        A, b = _spd(case, seed)
        x = torch.linalg.solve(A, b)
        x = x + torch.linalg.solve(A, b - A @ x)
        return {"x": x, "info": None}
    if kind == "budget" and not case["sgma"] and not case["mixed"]:
        return _exact_budgeted(case, seed)
    if kind != "predict":
        return None  # the weights where the iteration happened to stop: no value apart from the iteration's own
    X, y = _matrix(case, case["rows"] + case["vectors"], seed)
    beta = torch.from_numpy(_weights(y[case["rows"]:], 10.0, np.random.default_rng([seed, 7]))).cuda()
    X = torch.from_numpy(np.ascontiguousarray(X, dtype=np.float64)).cuda()
    T, S = X[:case["rows"]], X[case["rows"]:]
    K = T @ S.T
    if not case["linear"]:
        K = torch.exp(-GAMMA[case["data"]] * ((T * T).sum(1)[:, None] + (S * S).sum(1)[None, :] - 2.0 * K))
    f = K @ beta[:-1] + beta[-1]
    return f if case["soft"] else torch.where(f >= 0.0, 1.0, -1.0).double()
