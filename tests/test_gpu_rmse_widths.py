"""The squared-error kernel's load widths (f a multiple of 4, of 2, odd) and its special values,
against FP64 numpy."""
from __future__ import annotations

import numpy as np
import pytest

import cuda_als_gb300 as ca

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f", [1, 2, 3, 4, 6, 7, 8, 100, 127, 128])
@pytest.mark.parametrize("values", ["plain", "zeros", "subnormal", "nan"])
def test_rmse_load_widths_and_special_values(f, values):
    rng = np.random.default_rng(f)
    m, n, k = 300, 200, 5000
    U = (rng.standard_normal((m, f)) * 0.5).astype(np.float32)
    V = (rng.standard_normal((n, f)) * 0.5).astype(np.float32)
    if values == "zeros":
        U[::3] = 0.0
        V[:, f // 2] = -0.0
    if values == "subnormal":
        U[::2] = np.float32(1e-40)
        V[::3, 0] = np.float32(-3e-42)
    if values == "nan":
        U[5, f // 2:] = np.nan
        V[7, f - 1] = np.nan
    r, c = rng.integers(0, m, k).astype(np.int32), rng.integers(0, n, k).astype(np.int32)
    v = rng.integers(1, 6, k).astype(np.float32)
    tr = ca.host_sparse_matrix(m, n, 1).set_csr(np.r_[0, np.ones(m)].astype(np.int32), [0], [1.0])
    te = ca.host_sparse_matrix(m, n, k).set_coo(r, c, v)
    with ca.als_model(tr, te, f, 0.05, 1) as mdl:
        mdl.set_factors(U, V)
        got = mdl.rsme_test()
    p = U[r].astype(np.float64) * V[c].astype(np.float64)
    # the dot product ends before the first NaN component
    dead = np.cumsum(np.isnan(U[r]) | np.isnan(V[c]), axis=1) > 0
    pred = np.where(dead, 0.0, p).sum(axis=1)
    want = np.sqrt(np.mean((v.astype(np.float64) - pred) ** 2))
    assert got == pytest.approx(want, rel=1e-13)  # FP64 sums of at most 5,000 x 128 terms
