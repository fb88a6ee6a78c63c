"""Where the adjoint's gradient goes: pageable and page-locked memory, and a device array, which
the copy alone decides about (the host never writes to it)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import cuda_als_gb300 as ca
from conftest import random_csr
from cuda_als_gb300._lib import CsrView, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", ["pageable", "pinned", "device"])
def test_the_gradients_memory(where):
    torch = pytest.importorskip("torch")
    m, n, f = 40, 3000, 16
    ptr, idx, val = random_csr(np.random.default_rng(0), m, n, density=0.05)
    tr = ca.host_sparse_matrix(m, n, len(idx)).set_csr(ptr, idx, val)
    V = (np.random.default_rng(1).standard_normal((n, f)) * 0.3).astype(np.float32)
    rows, cols, vals = np.arange(m, dtype=np.int32), np.arange(m, dtype=np.int32) * 3, np.ones(m, np.float32)
    view = CsrView(m, n, m, C.c_void_p(rows.ctypes.data), C.c_void_p(cols.ctypes.data),
                   C.c_void_p(vals.ctypes.data))
    loss, dlam = C.c_double(), C.c_double()
    out = torch.zeros((n, f), dtype=torch.float32, device="cuda" if where == "device" else "cpu",
                      pin_memory=where == "pinned")
    torch.cuda.synchronize()
    with ca.als_model(tr, None, f, 0.05, 1, ca.CALCULATE_VTVS_TYPE.SIMPLE, ca.SOLVE_TYPE.CHOLESKY) as mdl:
        mdl.set_factors(None, V)
        want = mdl.user_halfsweep_adjoint(rows, cols, vals)[1]
        mdl.set_factors(None, V)
        status = lib().als_user_halfsweep_adjoint(mdl._h, C.byref(view), C.byref(loss),
                                                  C.c_void_p(out.data_ptr()), C.byref(dlam))
    torch.cuda.synchronize()
    if where == "device":
        assert status in (0, ca.Status.CUDA)
    else:
        assert status == 0
    if status == 0:
        assert np.array_equal(out.cpu().numpy(), want)
