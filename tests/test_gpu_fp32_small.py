"""FP32 rows at f <= 32: the CTA has a warp more where rows are few; a row's bits are the same either
way, and for every solver close to the FP64 oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import cuda_als_gb300 as ca
from conftest import random_csr
from oracle import oracle as O
from test_gpu_fp32_tiles import DEGREES, TOL_DIRECT, _users

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f", [1, 8, 9, 16, 17, 24, 25, 32])
@pytest.mark.parametrize("solve,osolve", [(ca.SOLVE_TYPE.LU, O.LU),
                                          (ca.SOLVE_TYPE.CHOLESKY, O.CHOLESKY)])
def test_few_and_many_rows_agree(f, solve, osolve):
    rng = np.random.default_rng(f)
    few, many, n = len(DEGREES), 8 * 152 + 1, 400
    ptr, idx, val = random_csr(rng, many, n, degrees=(DEGREES * (many // few + 1))[:many])
    V = (rng.standard_normal((n, f)) * 0.3).astype(np.float32)
    U = np.zeros((many, f), np.float32)
    X, flagged = _users(many, n, ptr, idx, val, f, 0.05, solve, U, V)
    k = int(ptr[few])
    Xf, _ = _users(few, n, ptr[:few + 1], idx[:k], val[:k], f, 0.05, solve, U[:few].copy(), V)
    assert flagged == 0 and np.array_equal(X[:few], Xf)
    Xe = U.copy()
    O.half_sweep(ptr, idx, val, V, Xe, f, 0.05, solve=osolve, cg_tol=0.0)
    err = np.linalg.norm(X.astype(np.float64) - Xe, axis=1)
    assert (err / np.maximum(np.linalg.norm(Xe, axis=1), 1e-6)).max() < TOL_DIRECT
