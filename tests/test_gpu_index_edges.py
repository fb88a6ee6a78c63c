"""The transposes and the triples builder at the edges of their tiles, digits and packed words:
bit-exact against numpy's stable sort."""
from __future__ import annotations

import numpy as np
import pytest

import cuda_als_gb300 as ca
from cuda_als_gb300._lib import lib
from test_zz_no_alloc import _transpose

pytestmark = pytest.mark.gpu


def _csr(rng, m, n, nnz):
    """nnz entries (cells may repeat) over few rows among many; columns from both ends of the range."""
    row = np.sort(rng.integers(0, m, nnz) // max(1, m // 64) * max(1, m // 64))
    col = np.where(rng.random(nnz) < 0.3, n - 1 - rng.integers(0, min(n, 3), nnz), rng.integers(0, n, nnz))
    ptr = np.zeros(m + 1, np.int64)
    np.add.at(ptr, row + 1, 1)
    return row, ptr.cumsum(), col, rng.integers(1, 11, nnz).astype(np.float32) / 2


# columns at a digit's and a pass's edge; 2^25 rows: row and column parts no longer share a word
@pytest.mark.parametrize("m,n", [(300, 1), (300, 2), (300, 256), (300, 257), (300, 65536),
                                 (300, 65537), (1, 5000), (1 << 24, 65536), ((1 << 25), 65536),
                                 ((1 << 25), 257)])
@pytest.mark.parametrize("nnz", [1, 4095, 4096, 4097, 40960])
def test_transposes_at_the_edges(m, n, nnz):
    torch = pytest.importorskip("torch")
    row, ptr, col, val = _csr(np.random.default_rng(nnz + n), m, n, nnz)
    order = np.argsort(col, kind="stable")
    want = np.concatenate([[0], np.bincount(col, minlength=n).cumsum()])
    for fn in (lib().als_csr_to_csc_device, lib().als_csr_to_csc_device_noalloc):
        status, cptr, ridx, cval = _transpose(fn, torch, m, n, ptr, col, val)
        assert status == 0
        assert np.array_equal(cptr, want)
        assert np.array_equal(ridx, row[order]) and np.array_equal(cval, val[order])


# 32 bits of row and column share a key, 33 do not; cells repeat across tiles of 4,096 entries
@pytest.mark.parametrize("m,n", [(1, 1), (3, 1), (1, 300), (1 << 17, 1 << 15), ((1 << 17) + 1, 1 << 15),
                                 (40, 1 << 27)])
@pytest.mark.parametrize("nnz", [1, 4096, 4097, 20000])
@pytest.mark.parametrize("cells", [1, 700])
def test_builder_at_the_edges(m, n, nnz, cells):
    rng = np.random.default_rng(nnz + cells)
    cr, cc = rng.integers(0, m, cells), rng.integers(0, n, cells)
    cr[0], cc[0] = m - 1, n - 1
    at = rng.integers(0, cells, nnz)
    val = rng.integers(1, 11, nnz).astype(np.float32) / 2
    key = cr[at] * n + cc[at]
    cell, inv = np.unique(key, return_inverse=True)
    total = np.bincount(inv, weights=val).astype(np.float32)
    (ptr, idx, v), rows, (cptr, ridx, cval) = ca.coo_to_csr(m, n, cr[at], cc[at], val)
    assert np.array_equal(rows, cell // n) and np.array_equal(idx, cell % n)
    assert np.array_equal(v, total)
    assert np.array_equal(ptr, np.searchsorted(cell // n, np.arange(m + 1)))
    order = np.argsort(cell % n, kind="stable")
    assert np.array_equal(cptr, np.searchsorted((cell % n)[order], np.arange(n + 1)))
    assert np.array_equal(ridx, (cell // n)[order]) and np.array_equal(cval, total[order])


def test_update_values_through_the_permutation():
    """A handle whose CSC was given: the first update builds the permutation (65,537 columns take
    three passes, 300 two), the second gathers by it."""
    for m, n in ((500, 300), (500, 65537)):
        row, ptr, col, val = _csr(np.random.default_rng(n), m, n, 9000)
        keep = np.unique(row * n + col, return_index=True)[1]
        row, col, val = row[keep], col[keep], val[keep]
        ptr = np.concatenate([[0], np.bincount(row, minlength=m).cumsum()])
        order = np.argsort(row * n + col, kind="stable")
        row, col, val = row[order], col[order], val[order]

        def matrix(v):
            t = ca.host_sparse_matrix(m, n, len(v))
            t.set_csr(ptr.astype(np.int32), col.astype(np.int32), v)
            return t

        def factors(mdl):
            mdl.init_factors()
            mdl.iterate(1)
            U, V = np.empty((m, 8), np.float32), np.empty((n, 8), np.float32)
            mdl.get_factors(U, V)
            return U, V

        def model(v):
            return ca.als_model(matrix(v), None, 8, 0.05, 1, ca.CALCULATE_VTVS_TYPE.SMEM_ROW_MAJOR, 3)

        mdl = model(val)
        for scale in (0.5, 2.0):
            new = (val * np.float32(scale)).astype(np.float32)
            mdl.update_values(new)
            got, want = factors(mdl), factors(model(new))
            assert all(np.array_equal(a, b) for a, b in zip(got, want))
