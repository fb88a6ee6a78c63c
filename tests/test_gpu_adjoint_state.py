"""What a handle keeps between adjoint calls (the item chunks, the workspace): every call's results are
those of a fresh handle, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import cuda_als_gb300 as ca

pytestmark = pytest.mark.gpu

M, N, F, LAM = 6000, 60, 24, 0.05


def _patterns():
    """Popular first items (several chunks of 2,048 ratings), then popular last ones: equal counts."""
    rng = np.random.default_rng(1)
    hit = rng.random((M, N)) < np.linspace(0.95, 0.01, N)[None, :] ** 2
    hit[::7] = False  # users without ratings
    for cells in (hit, hit[::-1, ::-1]):
        ptr = np.concatenate([[0], cells.sum(1).cumsum()]).astype(np.int32)
        val = rng.integers(1, 6, int(ptr[-1])).astype(np.float32)
        yield ca.host_sparse_matrix(M, N, int(ptr[-1])).set_csr(ptr, np.nonzero(cells)[1].astype(np.int32), val)


def _held(seed, k):
    rng = np.random.default_rng(seed)
    return [rng.integers(0, M, k).astype(np.int32), rng.integers(0, N, k).astype(np.int32),
            rng.integers(1, 6, k).astype(np.float32)]


def test_calls_on_one_handle_equal_a_fresh_ones():
    V = (np.random.default_rng(9).standard_normal((N, F)) * 0.3).astype(np.float32)
    Y = V.astype(np.float64) * (1.0 + 1e-9)

    def model(tr):
        return ca.als_model(tr, None, F, LAM, 1, ca.CALCULATE_VTVS_TYPE.SIMPLE, ca.SOLVE_TYPE.CHOLESKY)

    def adjoint(mdl, held, f64):
        if f64:
            return mdl.user_halfsweep_adjoint_f64(*held, Y, LAM)
        mdl.set_factors(None, V)
        return mdl.user_halfsweep_adjoint(*held)

    def fresh(tr, held, f64):
        with model(tr) as mdl:
            return adjoint(mdl, held, f64)

    first, second = _patterns()
    # held-out sets smaller and larger than before, and none; FP64's larger workspace, then FP32 in it
    calls = [(7, 400, False), (8, 30, False), (9, 0, False), (10, 9000, False), (11, 50, True),
             (12, 700, False), (13, 0, True)]
    with model(first) as mdl:
        for k, tr in enumerate((first, second, first)):
            if k:
                mdl.reload(tr)
            for seed, nh, f64 in calls:
                held = _held(seed, nh)
                got, want = adjoint(mdl, held, f64), fresh(tr, held, f64)
                assert got[0] == want[0] and got[2] == want[2] and np.array_equal(got[1], want[1])
                bad = _held(seed, 20)
                bad[1][7] = N
                with pytest.raises(ca.ALSError) as e:  # a refused call in between
                    mdl.user_halfsweep_adjoint(*bad)
                assert e.value.status == ca.Status.INVALID_ARG
