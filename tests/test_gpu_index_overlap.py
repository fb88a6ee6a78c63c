"""The transposes in place, and the triples builder with CSC outputs over its inputs."""
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

@pytest.mark.parametrize("m,n", [(3, 1), (300, 200), (9000, 9000), (1 << 17, 1 << 16)])
@pytest.mark.parametrize("nnz", [30000, 2000000])
@pytest.mark.parametrize("over", ["val", "all"])
def test_the_builder_with_csc_outputs_over_its_inputs(m, n, nnz, over):
    """csc_vals in the place of the triples' values, or also row_idxs in that of their rows."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    r, c = rng.integers(0, m, nnz).astype(np.int32), rng.integers(0, n, nnz).astype(np.int32)
    v = rng.integers(1, 11, nnz).astype(np.float32) / 2
    dev = torch.device("cuda", 0)

    def build(overlap):
        tr, tc, tv = (torch.from_numpy(a.copy()).to(dev) for a in (r, c, v))
        i32 = lambda k: torch.zeros(k, dtype=torch.int32, device=dev)  # noqa: E731
        f32 = lambda k: torch.zeros(k, dtype=torch.float32, device=dev)  # noqa: E731
        out = [i32(m + 1), i32(nnz), f32(nnz), i32(nnz), i32(n + 1),
               tr if overlap and over == "all" else i32(nnz), tv if overlap else f32(nnz)]
        view = CsrView(m, n, nnz, C.c_void_p(tr.data_ptr()), C.c_void_p(tc.data_ptr()),
                       C.c_void_p(tv.data_ptr()))
        k = C.c_int64()
        status = lib().als_coo_to_csr_device(C.byref(view), *[C.c_void_p(t.data_ptr()) for t in out], C.byref(k),
                                             C.c_void_p(torch.cuda.current_stream(dev).cuda_stream))
        assert status == 0, lib().als_last_error(None)
        torch.cuda.synchronize(dev)
        kk = k.value
        return [out[0], out[1][:kk], out[2][:kk], out[3][:kk], out[4], out[5][:kk], out[6][:kk]]

    for a, b in zip(build(False), build(True)):
        assert torch.equal(a, b)
