"""FP32 L D L^T at the ends of the exponent range, on matrices whose every operation is exact."""
from __future__ import annotations

import numpy as np
import pytest

import cuda_als_gb300 as ca

pytestmark = pytest.mark.gpu


def _model(f, d, r):
    """One user who rated every item; item j's factors are d_j e_j: A = diag(d_j^2), x_j = r_j / d_j."""
    tr = ca.host_sparse_matrix(1, f, f).set_csr(np.array([0, f], np.int32), np.arange(f, dtype=np.int32), r)
    mdl = ca.als_model(tr, None, f, 0.0, 1, ca.CALCULATE_VTVS_TYPE.SIMPLE, ca.SOLVE_TYPE.CHOLESKY,
                       precision=int(ca.PRECISION.FP32))
    mdl.set_factors(np.zeros((1, f), np.float32), np.diag(d).astype(np.float32))
    return mdl


# the tiles' last block has 1, 4 and 7 live columns of 8
@pytest.mark.parametrize("f", [1, 7, 12, 33, 100, 129, 175])
@pytest.mark.parametrize("e", [-66, -64, -63, 63])
def test_a_last_pivot_at_the_end_of_the_range(f, e):
    """Last pivots of 2^-132 and 2^-128 have infinite reciprocals in FP32: none of that reaches the
    solution, whose terms are powers of two times the ratings."""
    d = np.ones(f)
    d[-1] = 2.0 ** e
    r = (np.arange(f) % 5 + 1).astype(np.float32)
    with _model(f, d, r) as mdl:
        mdl.half_sweep(0)
        U, _ = mdl.get_factors()
        assert mdl.counters()["flagged_rows"] == 0
        assert np.array_equal(U[0].astype(np.float64), r / d)


@pytest.mark.parametrize("f", [1, 7, 12, 33, 100, 129, 175])
def test_the_adjoint_with_an_infinite_reciprocal(f):
    """The same matrix, a held-out rating of the last item 2^-20 above its prediction: g = A^-1 h has
    the one term -2^(-19 + 66)."""
    d = np.ones(f)
    d[-1] = 2.0 ** -66
    r = np.ones(f, np.float32)
    with _model(f, d, r) as mdl:
        loss, G, dlam = mdl.user_halfsweep_adjoint([0], [f - 1], [1.0 + 2.0 ** -20])
        U, _ = mdl.get_factors()
        assert mdl.counters()["flagged_rows"] == 0
    assert np.array_equal(U[0].astype(np.float64), 1.0 / d)
    g = -(2.0 ** 47)
    assert loss == 2.0 ** -40
    assert dlam == -f * g * 2.0 ** 66
    # dL/dy_i: (r - y_i . x) g - (g . y_i) x over the ratings (r = y_i . x), -2 (2^-20) x held out
    want = np.zeros((f, f))
    want[-1] = -(g * d[-1]) / d - 2.0 ** -19 / d
    assert np.array_equal(G.astype(np.float64), want)
