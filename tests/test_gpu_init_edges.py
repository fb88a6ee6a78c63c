"""als_init_factors against the C library's rand(), at the edges of a warp's and a CTA's calls."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import cuda_als_gb300 as ca

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,f", [(1, 1), (31, 1), (32, 31), (993, 1), (3968, 1), (3969, 1), (10677, 64)])
def test_init_is_srand_0(n, f):
    tr = ca.host_sparse_matrix(1, n, 1)
    tr.set_csr(np.array([0, 1], np.int32), np.array([0], np.int32), np.array([1.0], np.float32))
    mdl = ca.als_model(tr, None, f, 0.05, 1, ca.CALCULATE_VTVS_TYPE.SMEM_ROW_MAJOR, 3)
    mdl.init_factors()
    U, V = np.ones((1, f), np.float32), np.empty((n, f), np.float32)
    mdl.get_factors(U, V)
    libc = C.CDLL(None)
    libc.srand(0)
    r = np.array([libc.rand() for _ in range(n * f)], np.int32)
    want = (0.2 * (r.astype(np.float32) / np.float32(2147483647)).astype(np.float64)).astype(np.float32)
    assert np.array_equal(V.ravel(), want) and not U.any()
