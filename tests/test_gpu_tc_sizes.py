"""The solvers that stop at the row's last 16 features and the accumulators between the solver groups
(more of them the fewer features), at the sizes where either changes."""
from __future__ import annotations

import numpy as np
import pytest

import cuda_als_gb300 as ca
import test_gpu_tc as tc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f", [15, 17, 32, 33, 48, 49, 65, 80, 81, 96, 97, 112, 113])
def test_cholesky_at_every_last_block(f):
    tc.test_tc_half_sweep_matches_oracle_on_bf16_inputs(f)


@pytest.mark.parametrize("f", [17, 32, 33, 48, 49, 80, 81, 96, 97])
def test_fp16_gram_cg_between_accumulators(f):
    tc.test_tc_cg_fp16_runs_its_products_on_the_tensor_core(f)


@pytest.mark.parametrize("f", [10, 40, 100, 128])
def test_rows_without_a_factor_are_flagged_and_zero(f):
    """lambda = 0 and a feature that is zero in every item: its pivot is exactly zero."""
    rng, m, n, ptr, idx, val = tc.stage_boundary_problem(f)
    V0 = (rng.standard_normal((n, f)) * 0.3).astype(np.float32)
    V0[:, f // 2] = 0.0
    with tc.make_model(m, n, ptr, idx, val, f, lam=0.0) as mdl:
        mdl.set_factors(np.ones((m, f), np.float32), V0)
        mdl.half_sweep(0)
        U, _ = mdl.get_factors()
        assert mdl.counters()["flagged_rows"] == int((np.diff(ptr) > 0).sum())
    assert not U.any()
