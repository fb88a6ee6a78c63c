"""Work that users of this library have it do, as cases that can be timed and checked.

A case is one call (or the short run of calls a program makes) through a public entry point, at
sizes of the reference's datasets: the 1,000 x 500 toy sets, MovieLens 10M (69,878 x 10,677, 9.0M
training ratings), Netflix (480,189 x 17,770, 98.6M) and MovieLens latest (283,228 x 58,098,
24.3M).  Ratings are drawn on the GPU from a seed: lognormal row degrees, Zipf columns, distinct
cells, half-star values of planted factors plus noise.

kind "train"      als_model.train() from the srand(0) start, then the test RMSE
     "refresh"    a new rating snapshot into a living model: reload, init, one epoch, read back
     "half"       one half-sweep (side 0: users given items, 1: items given users) from planted
                  factors; the CG solvers start from the same warm start at every pass
     "adjoint"    held-out loss of the user half-sweep and its gradients
     "transpose"  CSR -> CSC on device arrays ("noalloc": the entry point that allocates nothing)
     "coo"        rating triples -> CSR, COO rows and CSC on device arrays
     "rmse"       the test RMSE of a trained model
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import cuda_als_gb300 as ca
from cuda_als_gb300._lib import CsrView, lib

LAM = 0.05
SOLVERS = {"lu": 0, "cg16": 1, "cg": 2, "chol": 3}
PRECISIONS = {"fp32": 0, "bf16": 1, "fp8": 2}
CG_STEPS, CG_TOL = 6, 1e-4  # the library's defaults


def listed():
    return [
        # the toy sets with the configuration defaults: a call that is launches and latency
        {"name": "train_toy_fp32_lu", "kind": "train", "m": 1000, "n": 500, "nnz": 18000,
         "test": 2000, "f": 10, "precision": "fp32", "solver": "lu", "iters": 10},
        # a nightly refresh of a MovieLens 10M model, end to end from host buffers
        {"name": "refresh_ml10m_bf16_chol", "kind": "refresh", "m": 69878, "n": 10677,
         "nnz": 9000000, "test": 1000000, "f": 64, "precision": "bf16", "solver": "chol"},
        # the default solver and precision (als_config_default: FP32 Gram, LU), users
        {"name": "users_ml10m_fp32_lu", "kind": "half", "m": 69878, "n": 10677, "nnz": 9000000,
         "f": 64, "precision": "fp32", "solver": "lu", "side": 0},
        # plain FP32 Cholesky on few, long rows (the accuracy baseline), items
        {"name": "items_netflix_fp32_chol", "kind": "half", "m": 480189, "n": 17770,
         "nnz": 98600000, "f": 100, "precision": "fp32", "solver": "chol", "side": 1},
        # the reference's CG on tensor-core Grams, many short rows
        {"name": "users_netflix_bf16_cg", "kind": "half", "m": 480189, "n": 17770,
         "nnz": 98600000, "f": 100, "precision": "bf16", "solver": "cg", "side": 0},
        # the reference's FP16-Gram CG, few long rows
        {"name": "items_netflix_bf16_cg16", "kind": "half", "m": 480189, "n": 17770,
         "nnz": 98600000, "f": 100, "precision": "bf16", "solver": "cg16", "side": 1},
        # Cholesky with refinement at the largest f of the tensor-core path
        {"name": "users_mllatest_bf16_chol", "kind": "half", "m": 283228, "n": 58098,
         "nnz": 24300000, "f": 128, "precision": "bf16", "solver": "chol", "side": 0},
        # FP8 operands where the Gram dominates: few long rows, f = 128
        {"name": "users_transposed_fp8_cg", "kind": "half", "m": 17770, "n": 480189,
         "nnz": 98600000, "f": 128, "precision": "fp8", "solver": "cg", "side": 0},
        # hyper-gradient step: backward through the user half-sweep
        {"name": "adjoint_mllatest_fp32", "kind": "adjoint", "m": 283228, "n": 58098,
         "nnz": 24300000, "held": 1000000, "f": 128, "dtype": "fp32"},
        # the transpose every new snapshot goes through
        {"name": "transpose_netflix", "kind": "transpose", "m": 480189, "n": 17770,
         "nnz": 98600000, "noalloc": False},
        # raw triples with some repeated cells, in no order
        {"name": "coo_ml10m", "kind": "coo", "m": 69878, "n": 10677, "nnz": 10000000},
        # evaluation after an iteration
        {"name": "rmse_netflix_test", "kind": "rmse", "m": 480189, "n": 17770, "nnz": 2000000,
         "test": 1408395, "f": 100},
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["train", "refresh", "half", "half", "half", "half", "adjoint",
                       "transpose", "coo", "rmse"])
    if kind == "train":
        m, n = logint(300, 3000), logint(200, 1500)
        return {"kind": kind, "m": m, "n": n, "nnz": int(m * n * rng.uniform(0.02, 0.1)),
                "test": logint(100, 4000), "f": rng.randint(4, 40), "precision": "fp32",
                "solver": rng.choice(["lu", "chol"]), "iters": rng.randint(1, 10)}
    if kind == "refresh":
        m, n = logint(2000, 70000), logint(500, 11000)
        return {"kind": kind, "m": m, "n": n, "nnz": min(9000000, int(m * n * 0.02), 150 * m),
                "test": logint(1000, 1000000), "f": rng.randint(16, 64), "precision": "bf16",
                "solver": "chol"}
    if kind == "half":
        prec = rng.choice(["fp32", "bf16", "bf16", "fp8"])
        solver = rng.choice(["lu", "chol", "cg"] if prec == "fp32" else
                            ["cg", "cg", "cg16", "chol"])
        m, n = logint(1000, 100000 if prec == "fp32" else 480189), logint(500, 58098)
        if rng.random() < 0.25:
            m, n = n, m
        f = rng.randint(8, 140) if prec == "fp32" else rng.randint(8, 128)
        # a row's work in the direct solvers grows with f cubed: fewer rows there
        nnz = min(int(m * n * rng.uniform(0.005, 0.08)), logint(20000, 20000000))
        return {"kind": kind, "m": m, "n": n, "nnz": max(nnz, m, n), "f": f, "precision": prec,
                "solver": solver, "side": rng.randint(0, 1)}
    if kind == "adjoint":
        f64 = rng.random() < 0.25
        m, n = logint(500, 2000 if f64 else 200000), logint(300, 1000 if f64 else 40000)
        nnz = min(int(m * n * rng.uniform(0.005, 0.05)), 20000000)
        return {"kind": kind, "m": m, "n": n, "nnz": max(nnz, m, n),
                "held": logint(200, 2000 if f64 else 1000000),
                "f": rng.randint(8, 32 if f64 else 128), "dtype": "fp64" if f64 else "fp32"}
    if kind == "transpose":
        noalloc = rng.random() < 0.4
        m, n = logint(100, 480189), logint(100, 480189)
        hi = 590000 if noalloc else 98600000
        return {"kind": kind, "m": m, "n": n, "nnz": min(int(m * n * 0.2), logint(2000, hi)),
                "noalloc": noalloc}
    if kind == "coo":
        m, n = logint(200, 283228), logint(100, 58098)
        return {"kind": kind, "m": m, "n": n,
                "nnz": min(int(m * n * 0.2), logint(2000, 30000000))}
    return {"kind": "rmse", "m": logint(1000, 480189), "n": logint(500, 58098),
            "nnz": 60000, "test": logint(1000, 1400000), "f": rng.randint(8, 128)}


# ------------------------------------------------------------------------------------- inputs


def _gen(seed, tag):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * (seed + 1) + tag)
    return g


def _cells(m, n, nnz, seed, tag):
    """nnz distinct (row, column) cells in row-major order: rows by lognormal weights, columns by
    Zipf weights in a random order."""
    g = _gen(seed, tag)
    rw = torch.randn(m, device="cuda", generator=g).mul_(1.0).exp_().double().cumsum(0)
    rank = torch.randperm(n, device="cuda", generator=g).double() + 1.0
    cw = (rank + 10.0).pow(-0.9).cumsum(0)
    keys = torch.empty(0, dtype=torch.int64, device="cuda")
    while keys.numel() < nnz:
        k = int((nnz - keys.numel()) * 1.25) + 1000
        r = torch.searchsorted(rw, torch.rand(k, device="cuda", generator=g,
                                              dtype=torch.float64) * rw[-1]).clamp_(max=m - 1)
        c = torch.searchsorted(cw, torch.rand(k, device="cuda", generator=g,
                                              dtype=torch.float64) * cw[-1]).clamp_(max=n - 1)
        keys = torch.unique(torch.cat([keys, r * n + c]))
        del r, c
    if keys.numel() > nnz:
        drop = torch.randperm(keys.numel(), device="cuda", generator=g)[: keys.numel() - nnz]
        keep = torch.ones(keys.numel(), dtype=torch.bool, device="cuda")
        keep[drop] = False
        keys = keys[keep]
    row = torch.div(keys, n, rounding_mode="floor")
    return row.int(), (keys - row * n).int()


def _factors(rows, f, seed, tag):
    a = math.sqrt(3.5 / f)
    return torch.randn(rows, f, device="cuda", generator=_gen(seed, tag)).mul_(0.6 * a).add_(a)


def _values(row, col, U, V, seed, tag):
    """Half-star ratings of the planted factors plus noise."""
    val = torch.randn(row.numel(), device="cuda", generator=_gen(seed, tag)).mul_(0.7)
    for b in range(0, row.numel(), 1 << 22):
        e = min(row.numel(), b + (1 << 22))
        val[b:e] += (U[row[b:e].long()] * V[col[b:e].long()]).sum(1)
    return val.mul_(2).round_().div_(2).clamp_(0.5, 5.0)


def _ptrs(idx, count):
    p = torch.zeros(count + 1, dtype=torch.int64, device="cuda")
    p[1:] = torch.bincount(idx, minlength=count).cumsum(0)
    return p.int()


def _problem(case, seed):
    """Planted factors, training CSR (row, ptr, col, val) and held-out triples, on the GPU."""
    m, n, f = case["m"], case["n"], case["f"]
    U, V = _factors(m, f, seed, 1), _factors(n, f, seed, 2)
    row, col = _cells(m, n, case["nnz"], seed, 3)
    val = _values(row, col, U, V, seed, 4)
    held = case.get("test", case.get("held", 0))
    hr = hc = hv = None
    if held:
        g = _gen(seed, 5)
        pick = torch.randint(case["nnz"], (held,), device="cuda", generator=g).sort().values
        hr = row[pick]
        hc = torch.randint(n, (held,), device="cuda", generator=g).int()
        hv = _values(hr, hc, U, V, seed, 6)
    return {"U": U, "V": V, "row": row, "ptr": _ptrs(row, m), "col": col, "val": val,
            "hr": hr, "hc": hc, "hv": hv}


def _perturbed(T, seed, tag):
    """Factors as they stand before a later epoch: near the planted ones."""
    f = T.shape[1]
    return T + torch.randn(T.shape, device="cuda",
                           generator=_gen(seed, tag)) * (0.15 * math.sqrt(3.5 / f))


def _matrices(case, P, pinned=False):
    tr = ca.host_sparse_matrix(case["m"], case["n"], case["nnz"], pinned)
    tr.set_csr(P["ptr"].cpu().numpy(), P["col"].cpu().numpy(), P["val"].cpu().numpy())
    te = None
    if P["hr"] is not None and case["kind"] != "adjoint":
        te = ca.host_sparse_matrix(case["m"], case["n"], P["hr"].numel(), pinned)
        te.set_coo(P["hr"].cpu().numpy(), P["hc"].cpu().numpy(), P["hv"].cpu().numpy())
    return tr, te


def _model(case, tr, te, iters=1):
    return ca.als_model(tr, te, case["f"], LAM, iters, ca.CALCULATE_VTVS_TYPE.SMEM_ROW_MAJOR,
                        SOLVERS[case.get("solver", "chol")],
                        precision=PRECISIONS[case.get("precision", "fp32")])


class _Device:
    """A float32 array that the model owns on the GPU, for torch.as_tensor (no copy); the tensor
    keeps this object, and it the model."""

    def __init__(self, model, ptr, shape):
        self.model = model
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "version": 3,
                                         "data": (ptr, False)}


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("transpose", "coo"):
        return _prepare_index(case, seed)
    P = _problem(case, seed)
    if kind == "refresh":  # the model lives on another snapshot of the same sizes
        old = dict(P, val=_values(P["row"], P["col"], P["U"], P["V"], seed, 7))
        model = _model(case, *_matrices(case, old))
        tr, te = _matrices(case, P, pinned=True)
        U, V = (np.empty((case[k], case["f"]), np.float32) for k in ("m", "n"))
        return {"kind": kind, "model": model, "train": tr, "test": te, "U": U, "V": V}
    tr, te = _matrices(case, P)
    model = _model(case, tr, te, case.get("iters", 1))
    state = {"kind": kind, "model": model}
    if kind == "train":
        return state
    U0, V0 = _perturbed(P["U"], seed, 8), _perturbed(P["V"], seed, 9)
    torch.cuda.synchronize()
    u, v = model.device_factors()
    dev = [torch.as_tensor(_Device(model, p, tuple(t.shape)), device="cuda")
           for p, t in ((u, U0), (v, V0))]
    dev[0].copy_(U0)
    dev[1].copy_(V0)
    if kind == "half":
        state["side"] = case["side"]
        state["X"] = dev[case["side"]]
        state["warm"] = (U0, V0)[case["side"]] if case["solver"] in ("cg", "cg16") else None
        state["stream"] = torch.cuda.Stream()
        model.set_stream(state["stream"].cuda_stream)
    if kind == "adjoint":
        state["held"] = tuple(P[k].cpu().numpy() for k in ("hr", "hc", "hv"))
        state["Y"] = V0.double().cpu().numpy() if case["dtype"] == "fp64" else None
    torch.cuda.synchronize()
    return state


def _prepare_index(case, seed):
    m, n, nnz = case["m"], case["n"], case["nnz"]
    i32 = dict(dtype=torch.int32, device="cuda")
    g = _gen(seed, 11)
    state = {"kind": case["kind"], "m": m, "n": n, "nnz": nnz, "stream": torch.cuda.Stream()}
    if case["kind"] == "transpose":
        row, col = _cells(m, n, nnz, seed, 3)
        state["in"] = (_ptrs(row, m), col,
                       torch.randint(1, 11, (nnz,), device="cuda", generator=g).float() / 2)
        state["out"] = (torch.empty(n + 1, **i32), torch.empty(nnz, **i32),
                        torch.empty(nnz, device="cuda"))
        state["noalloc"] = case["noalloc"]
    else:
        base = max(1, int(nnz * 0.99))  # one triple in a hundred repeats a cell
        row, col = _cells(m, n, base, seed, 3)
        at = torch.cat([torch.arange(base, device="cuda"),
                        torch.randint(base, (nnz - base,), device="cuda", generator=g)])
        at = at[torch.randperm(nnz, device="cuda", generator=g)]
        state["in"] = (row[at], col[at],
                       torch.randint(1, 11, (nnz,), device="cuda", generator=g).float() / 2)
        state["out"] = (torch.empty(m + 1, **i32), torch.empty(nnz, **i32),
                        torch.empty(nnz, device="cuda"), torch.empty(nnz, **i32),
                        torch.empty(n + 1, **i32), torch.empty(nnz, **i32),
                        torch.empty(nnz, device="cuda"))
    torch.cuda.synchronize()
    return state


# --------------------------------------------------------------------------------------- a pass


def _ok(status):
    if status:
        raise RuntimeError((lib().als_last_error(None) or b"").decode())


def run(state):
    kind = state["kind"]
    if kind == "transpose":
        view = CsrView(state["m"], state["n"], state["nnz"], *[t.data_ptr() for t in state["in"]])
        fn = lib().als_csr_to_csc_device_noalloc if state["noalloc"] else lib().als_csr_to_csc_device
        _ok(fn(C.byref(view), *[C.c_void_p(t.data_ptr()) for t in state["out"]],
               C.c_void_p(state["stream"].cuda_stream)))
        return state["out"]
    if kind == "coo":
        view = CsrView(state["m"], state["n"], state["nnz"], *[t.data_ptr() for t in state["in"]])
        count = C.c_int64()
        _ok(lib().als_coo_to_csr_device(C.byref(view),
                                        *[C.c_void_p(t.data_ptr()) for t in state["out"]],
                                        C.byref(count), C.c_void_p(state["stream"].cuda_stream)))
        k = count.value
        ptr, idx, val, row, cptr, ridx, cval = state["out"]
        return ptr, idx[:k], val[:k], row[:k], cptr, ridx[:k], cval[:k]
    model = state["model"]
    if kind == "train":
        model.train()
        return model.h_UT, model.h_VT, model.rsme_test()
    if kind == "refresh":
        model.reload(state["train"], state["test"])
        model.init_factors()
        model.iterate(1)
        model.get_factors(state["U"], state["V"])
        return state["U"], state["V"], model.rsme_test()
    if kind == "rmse":
        return model.rsme_test()
    if kind == "adjoint":
        if state["Y"] is not None:
            return model.user_halfsweep_adjoint_f64(*state["held"], state["Y"], LAM)
        return model.user_halfsweep_adjoint(*state["held"])
    if state["warm"] is not None:
        with torch.cuda.stream(state["stream"]):
            state["X"].copy_(state["warm"])
    model.half_sweep(state["side"])
    return state["X"]


def work(case):
    m, n, nnz, kind = case["m"], case["n"], case["nnz"], case["kind"]
    if kind == "transpose":
        return {"bytes": 16 * nnz + 4 * (m + n), "flops": 0}
    if kind == "coo":
        return {"bytes": 12 * nnz + 20 * nnz + 4 * (m + n), "flops": 0}
    f = case["f"]
    if kind == "rmse":
        t = case["test"]
        return {"bytes": 12 * t + 4 * f * (min(m, t) + min(n, t)), "flops": 2 * t * f}
    item = 8 if case.get("dtype") == "fp64" else 4
    solve = {"chol": f ** 3 / 3, "lu": 2 * f ** 3 / 3}.get(case.get("solver", "chol"),
                                                          2 * f * f * (CG_STEPS + 1))
    gram = nnz * (f * (f + 1) + 2 * f)
    if kind == "half":
        rows = (m, n)[case["side"]]
        warm = rows if case["solver"] in ("cg", "cg16") else 0
        return {"bytes": 8 * nnz + 4 * f * (m + n + warm), "flops": gram + rows * solve}
    if kind == "adjoint":
        return {"bytes": 16 * nnz + 2 * 12 * case["held"] + 2 * item * f * (m + n),
                "flops": gram + m * (solve + 8 * f * f) + 8 * f * nnz + 6 * f * case["held"]}
    iters = case.get("iters", 1)
    return {"bytes": iters * (16 * nnz + 8 * f * (m + n)) + 12 * case["test"] +
            (8 * nnz if kind == "refresh" else 0),
            "flops": iters * (2 * gram + (m + n) * solve) + 2 * f * case["test"]}


# ------------------------------------------------------------------------------ in 64 bits


def _solve64(ptr, idx, val, Y, n_out, case, X0=None, need=None):
    """Every row's solution in 64 bits, rows of near degrees in one batch; `need` receives each
    batch's (rows, entries, mask, Gram) as well."""
    f = Y.shape[1]
    deg = (ptr[1:] - ptr[:-1]).long()
    order = torch.argsort(deg, descending=True)
    X = torch.zeros(n_out, f, dtype=torch.float64, device="cuda")
    deg_host = deg[order].cpu().numpy()
    start, eye = 0, torch.eye(f, dtype=torch.float64, device="cuda")
    Yd = torch.cat([Y.double(), torch.zeros(1, f, dtype=torch.float64, device="cuda")])
    budget = (1 << 28) // f
    while start < n_out and deg_host[start] > 0:
        d = int(deg_host[start])
        stop = min(n_out, start + max(1, min(budget // d, (1 << 27) // (f * f))))
        low = int(np.searchsorted(-deg_host, -0.8 * d, side="right"))  # padding: a quarter at most
        stop = max(start + 1, min(stop, max(low, start + 64)))
        stop = min(stop, int(np.searchsorted(-deg_host, 0, side="left")))
        rows = order[start:stop]
        A = torch.zeros(len(rows), f, f, dtype=torch.float64, device="cuda")
        b = torch.zeros(len(rows), f, dtype=torch.float64, device="cuda")
        for k0 in range(0, d, budget):
            k = torch.arange(k0, min(d, k0 + budget), device="cuda")
            live = k[None, :] < deg[rows][:, None]
            at = (ptr[rows].long()[:, None] + k[None, :]).clamp_(max=idx.numel() - 1)
            Yr = Yd[torch.where(live, idx[at].long(), Y.shape[0])]
            A.baddbmm_(Yr.transpose(1, 2), Yr)
            b += torch.bmm(Yr.transpose(1, 2), torch.where(live, val[at].double(),
                                                           0.0).unsqueeze(2)).squeeze(2)
            del Yr
        A += (LAM * deg[rows].double())[:, None, None] * eye
        if case.get("solver") == "cg16":
            mant, ex = torch.frexp(A)
            A = torch.ldexp((mant * 2048).round() / 2048, ex)
        if case.get("solver") in ("cg", "cg16"):
            X[rows] = _cg64(A, b, X0[rows].double())
        else:
            L = torch.linalg.cholesky(A)
            X[rows] = torch.cholesky_solve(b.unsqueeze(2), L).squeeze(2)
            if need is not None:
                need(rows, L, X)
        start = stop
    return X


def _cg64(A, b, x):
    def mul(v):
        return torch.bmm(A, v.unsqueeze(2)).squeeze(2)

    r = b - mul(x)
    p, rs = r.clone(), (r * r).sum(1)
    live = torch.ones_like(rs, dtype=torch.bool)
    for _ in range(CG_STEPS):
        ap = mul(p)
        pap = (p * ap).sum(1)
        live = live & (pap > 0)
        alpha = torch.where(live, rs / pap, 0.0)
        x = x + alpha[:, None] * p
        r = r - alpha[:, None] * ap
        new = (r * r).sum(1)
        live = live & (new >= CG_TOL)
        p = r + (new / rs)[:, None] * p
        rs = new
    return x


def _rounded(T, precision):
    """The factor table as the path's operands hold it."""
    if precision == "bf16":
        return T.bfloat16().float()
    if precision == "fp8":  # one power of two per feature, the largest magnitude at most 448
        big = T.abs().amax(0).double()
        e = torch.ceil(torch.log2(big / 448.0))
        d = torch.exp2(e).float()
        return (T / d).to(torch.float8_e4m3fn).float() * d
    return T


def _columns(P, case):
    """The same ratings by column."""
    order = torch.argsort(P["col"], stable=True)
    return _ptrs(P["col"], case["n"]), P["row"][order], P["val"][order]


def _start64(count):
    """0.2 rand() / RAND_MAX after srand(0), as glibc's additive feedback generator gives it."""
    r = [1]
    for i in range(1, 31):
        r.append(16807 * r[-1] % 2147483647)
    r += r[:3]
    for i in range(34, 344 + count):
        r.append((r[i - 31] + r[i - 3]) & 0xffffffff)
    q = np.array([x >> 1 for x in r[344:]], np.float32) / np.float32(2147483648.0)
    return (0.2 * q.astype(np.float64)).astype(np.float32)


def _rmse64(U, V, P):
    s = 0.0
    for b in range(0, P["hr"].numel(), 1 << 20):
        r, c = P["hr"][b:b + (1 << 20)].long(), P["hc"][b:b + (1 << 20)].long()
        e = P["hv"][b:b + (1 << 20)].double() - (U[r].double() * V[c].double()).sum(1)
        s += float((e * e).sum())
    return math.sqrt(s / P["hr"].numel())


def exact(case, seed):
    kind = case["kind"]
    if kind == "transpose":  # whole numbers and copies of values
        return None
    if kind == "coo":
        return None
    P = _problem(case, seed)
    m, n, f = case["m"], case["n"], case["f"]
    prec = case.get("precision", "fp32")
    if kind in ("train", "refresh"):
        cp, ci, cv = _columns(P, case)
        V = torch.from_numpy(_start64(n * f).reshape(n, f)).cuda()
        for _ in range(case.get("iters", 1)):
            Y = _rounded(V.float(), prec) if prec != "fp32" else V
            U = _solve64(P["ptr"], P["col"], P["val"], Y, m, case)
            Y = _rounded(U.float(), prec) if prec != "fp32" else U
            V = _solve64(cp, ci, cv, Y, n, case)
        return U, V, _rmse64(U, V, P)
    U0, V0 = _perturbed(P["U"], seed, 8), _perturbed(P["V"], seed, 9)
    if kind == "rmse":
        return _rmse64(U0, V0, P)
    if kind == "half":
        if case["side"] == 0:
            return _solve64(P["ptr"], P["col"], P["val"], _rounded(V0, prec), m, case, U0)
        return _solve64(*_columns(P, case), _rounded(U0, prec), n, case, V0)
    # adjoint: the held-out residuals' gradient through every row's solution
    hr, hc, hv = P["hr"].long(), P["hc"].long(), P["hv"].double()
    Y = V0.double()
    G = torch.zeros(m, f, dtype=torch.float64, device="cuda")
    hptr = _ptrs(P["hr"], m).long()
    sums = {"loss": 0.0}

    def back(rows, L, X):
        count = hptr[rows + 1] - hptr[rows]
        at = torch.repeat_interleave(hptr[rows] - (count.cumsum(0) - count), count) + \
            torch.arange(int(count.sum()), device="cuda")
        which = torch.repeat_interleave(torch.arange(len(rows), device="cuda"), count)
        h = torch.zeros(len(rows), f, dtype=torch.float64, device="cuda")
        res = hv[at] - (X[rows][which] * Y[hc[at]]).sum(1)
        h.index_add_(0, which, -2.0 * res[:, None] * Y[hc[at]])
        G[rows] = torch.cholesky_solve(h.unsqueeze(2), L).squeeze(2)

    X = _solve64(P["ptr"], P["col"], P["val"], Y, m, case, need=back)
    dY = torch.zeros(n, f, dtype=torch.float64, device="cuda")
    for b in range(0, case["nnz"], 1 << 21):
        r, c = P["row"][b:b + (1 << 21)].long(), P["col"][b:b + (1 << 21)].long()
        x, g, y = X[r], G[r], Y[c]
        e = P["val"][b:b + (1 << 21)].double() - (x * y).sum(1)
        dY.index_add_(0, c, e[:, None] * g - (g * y).sum(1, keepdim=True) * x)
    for b in range(0, hr.numel(), 1 << 21):
        x, y = X[hr[b:b + (1 << 21)]], Y[hc[b:b + (1 << 21)]]
        res = hv[b:b + (1 << 21)] - (x * y).sum(1)
        sums["loss"] += float((res * res).sum())
        dY.index_add_(0, hc[b:b + (1 << 21)], -2.0 * res[:, None] * x)
    deg = (P["ptr"][1:] - P["ptr"][:-1]).double()
    return sums["loss"], dY, -float((deg * (G * X).sum(1)).sum())
