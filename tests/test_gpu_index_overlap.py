"""The transposes in place."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from cuda_als_gb300._lib import CsrView, lib
from test_gpu_index_edges import _csr

pytestmark = pytest.mark.gpu


# one, two and three passes of packed words; rows and columns that share no word
@pytest.mark.parametrize("m,n", [(300, 200), (300, 257), (300, 65536), (300, 65537), (1 << 25, 65536)])
@pytest.mark.parametrize("nnz", [1, 4097, 40960, 4000000])
@pytest.mark.parametrize("entry", ["als_csr_to_csc_device", "als_csr_to_csc_device_noalloc"])
def test_a_transpose_in_place(m, n, nnz, entry):
    torch = pytest.importorskip("torch")
    if entry.endswith("noalloc"):
        nnz = min(nnz, 593856)  # the most it takes
    row, ptr, col, val = _csr(np.random.default_rng(nnz + n), m, n, nnz)
    dev = torch.device("cuda", 0)
    for ids_only in (False, True):
        d_ptr = torch.from_numpy(ptr.astype(np.int32)).to(dev)
        d_idx = torch.from_numpy(col.astype(np.int32)).to(dev)
        d_val = torch.from_numpy(val).to(dev)
        o_ptr = torch.full((n + 1,), -7, dtype=torch.int32, device=dev)
        o_val = torch.empty_like(d_val) if ids_only else d_val
        view = CsrView(m, n, nnz, d_ptr.data_ptr(), d_idx.data_ptr(), d_val.data_ptr())
        stream = torch.cuda.current_stream(dev)
        status = getattr(lib(), entry)(C.byref(view), C.c_void_p(o_ptr.data_ptr()),
                                       C.c_void_p(d_idx.data_ptr()), C.c_void_p(o_val.data_ptr()),
                                       C.c_void_p(stream.cuda_stream))
        assert status == 0, lib().als_last_error(None)
        torch.cuda.synchronize(dev)
        order = np.argsort(col, kind="stable")
        assert np.array_equal(o_ptr.cpu().numpy(),
                              np.concatenate([[0], np.bincount(col, minlength=n).cumsum()]))
        assert np.array_equal(d_idx.cpu().numpy(), row[order])
        assert np.array_equal(o_val.cpu().numpy(), val[order])
