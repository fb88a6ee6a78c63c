"""The FP32 kernels that keep a row's matrix in registers (f <= 175) at the edges of their tiles,
panels and rating chunks, against the FP64 oracle; the wide kernels just above; the reciprocals of
pivots outside the normal range; the adjoint at the same edges."""
from __future__ import annotations

import numpy as np
import pytest

import cuda_als_gb300 as ca
from conftest import random_csr
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# 8 columns a tile, panel pitches 32 / 64 / 128 / 192, the last register size and the first above
SIZES = [1, 7, 8, 9, 31, 33, 64, 65, 72, 101, 128, 129, 174, 175, 176]
# ratings: around the 16-rating ring slots and the 32-rating right-hand-side sums
DEGREES = [1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 64, 65, 200, 0, 3]
# a row's error is within a few u cond(A); cond <= (0.09 f + lambda) / lambda = 320 at f = 176
# (one rating), u = 6e-8: 10 u cond
TOL_DIRECT = 2e-4
TOL_CG = 1e-3


def _problem(f, scale=0.3):
    rng = np.random.default_rng(f)
    m, n = len(DEGREES), 400
    ptr, idx, val = random_csr(rng, m, n, degrees=DEGREES)
    V = (rng.standard_normal((n, f)) * scale).astype(np.float32)
    U = (rng.standard_normal((m, f)) * 0.1).astype(np.float32)
    return m, n, ptr, idx, val, U, V


def _users(m, n, ptr, idx, val, f, lam, solve, U, V):
    tr = ca.host_sparse_matrix(m, n, len(idx)).set_csr(ptr, idx, val)
    with ca.als_model(tr, None, f, lam, 1, ca.CALCULATE_VTVS_TYPE.SIMPLE, solve,
                      precision=int(ca.PRECISION.FP32), cg_tol=0.0) as mdl:
        mdl.set_factors(U, V)
        mdl.half_sweep(0)
        return mdl.get_factors()[0], mdl.counters()["flagged_rows"]


@pytest.mark.parametrize("f", SIZES)
@pytest.mark.parametrize("solve,osolve,tol", [
    (ca.SOLVE_TYPE.LU, O.LU, TOL_DIRECT), (ca.SOLVE_TYPE.CHOLESKY, O.CHOLESKY, TOL_DIRECT),
    (ca.SOLVE_TYPE.CUMF_ALS_CG_FP32, O.CG_FP32, TOL_CG)])
def test_tile_edges_match_the_oracle(f, solve, osolve, tol):
    m, n, ptr, idx, val, U, V = _problem(f)
    X, flagged = _users(m, n, ptr, idx, val, f, 0.05, solve, U, V)
    Xe = U.copy()
    O.half_sweep(ptr, idx, val, V, Xe, f, 0.05, solve=osolve, cg_tol=0.0)
    err = np.linalg.norm(X.astype(np.float64) - Xe, axis=1)
    assert (err / np.maximum(np.linalg.norm(Xe, axis=1), 1e-6)).max() < tol
    assert flagged == 0 and not X[DEGREES.index(0)].any()


@pytest.mark.parametrize("f", [8, 37, 100])
@pytest.mark.parametrize("solve", [ca.SOLVE_TYPE.LU, ca.SOLVE_TYPE.CHOLESKY])
def test_tiny_pivots_scale_exactly(f, solve):
    """Factors scaled by 2^-55 put every pivot below 2^-100, where reciprocals are divisions; with
    lambda = 0 each operation scales by a power of two, so the solution scales exactly."""
    rng = np.random.default_rng(f)
    m, n = 6, 600
    ptr, idx, val = random_csr(rng, m, n, degrees=[600, 500, 400, 333, 320, 599])
    V = (rng.standard_normal((n, f)) * 0.3).astype(np.float32)
    U = np.zeros((m, f), np.float32)
    X, flagged = _users(m, n, ptr, idx, val, f, 0.0, solve, U, V)
    Xs, flagged_s = _users(m, n, ptr, idx, val, f, 0.0, solve, U, V * np.float32(2.0 ** -55))
    assert flagged == 0 and flagged_s == 0
    assert np.array_equal(Xs, X * np.float32(2.0 ** 55))


@pytest.mark.parametrize("solve", [ca.SOLVE_TYPE.LU, ca.SOLVE_TYPE.CHOLESKY])
@pytest.mark.parametrize("bad", [0.0, np.inf, np.nan])
def test_unsolvable_rows_are_zero_and_counted(solve, bad):
    """A zero, infinite or NaN Gram: x = 0, the row counted, its neighbours untouched."""
    f = 20
    m, n, ptr, idx, val, U, V = _problem(f)
    V[idx[ptr[13]:ptr[13 + 1]]] = 0.0 if bad == 0.0 else V[idx[ptr[13]:ptr[13 + 1]]]
    only = ptr[13] + np.arange(3)
    if bad != 0.0:
        V[idx[only[0]], 5] = bad
    lam = 0.0 if bad == 0.0 else 0.05
    keep = np.array([ptr[13], ptr[13 + 1]]) - ptr[13]
    X, flagged = _users(1, n, keep.astype(np.int32), idx[ptr[13]:ptr[14]], val[ptr[13]:ptr[14]], f,
                        lam, solve, U[:1], V)
    assert flagged == 1 and not X.any()


@pytest.mark.parametrize("f", [7, 33, 65, 129, 175, 176])
def test_adjoint_tile_edges(f):
    m, n, ptr, idx, val, U, V = _problem(f)
    rng = np.random.default_rng(1000 + f)
    held = (np.sort(rng.integers(0, m, 60)).astype(np.int32),
            rng.integers(0, n, 60).astype(np.int32),
            rng.integers(1, 6, 60).astype(np.float32))
    lam = float(np.float32(0.05))
    tr = ca.host_sparse_matrix(m, n, len(idx)).set_csr(ptr, idx, val)
    with ca.als_model(tr, None, f, lam, 1, ca.CALCULATE_VTVS_TYPE.SIMPLE,
                      ca.SOLVE_TYPE.CHOLESKY) as mdl:
        mdl.set_factors(None, V)
        loss, G, dlam = mdl.user_halfsweep_adjoint(*held)
    e_loss, _, e_G, e_dlam = O.user_adjoint(m, n, f, lam, (ptr, idx, val), V, held)
    assert loss == pytest.approx(e_loss, rel=1e-4)
    assert np.linalg.norm(G - e_G) / np.linalg.norm(e_G) < 2e-3
    assert dlam == pytest.approx(e_dlam, rel=5e-3)
