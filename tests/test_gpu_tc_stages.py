"""The tensor-core sweep's stage pipeline at its edges: rows of exactly and about a stage, a batch of
descriptors (32 stages published at once) and more than the descriptor and operand rings hold, at
the padded sizes' boundaries, against the FP64 oracle on the rounded table."""
from __future__ import annotations

import numpy as np
import pytest

import cuda_als_gb300 as ca
from conftest import random_csr
from oracle import oracle as O
from oracle import quant
from test_gpu_tc import TOL_BF16_INPUTS, bf16_round, make_model, rel_rows

pytestmark = pytest.mark.gpu

DEGREES = [1, 0, 63, 64, 65, 127, 128, 129, 31 * 64, 32 * 64, 32 * 64 + 1, 33 * 64 - 1, 64 * 64,
           64 * 64 + 17, 5000, 2, 0, 48, 16, 17]


@pytest.mark.parametrize("precision", [ca.PRECISION.BF16, ca.PRECISION.FP8])
@pytest.mark.parametrize("f", [8, 32, 33, 64, 65, 112, 113, 128])
@pytest.mark.parametrize("solve", [ca.SOLVE_TYPE.CHOLESKY, ca.SOLVE_TYPE.CUMF_ALS_CG_FP32])
def test_long_rows_and_descriptor_batches(f, precision, solve):
    rng = np.random.default_rng(f)
    m, n = len(DEGREES), 5200
    ptr, idx, val = random_csr(rng, m, n, degrees=DEGREES)
    U0 = (rng.standard_normal((m, f)) * 0.1).astype(np.float32)
    V0 = (rng.standard_normal((n, f)) * 0.3).astype(np.float32)
    with make_model(m, n, ptr, idx, val, f, solve=solve, precision=int(precision),
                    cg_tol=0.0) as mdl:
        mdl.set_factors(U0, V0)
        mdl.half_sweep(0)
        U, _ = mdl.get_factors()
        assert mdl.counters()["flagged_rows"] == 0
    Y = bf16_round(V0) if precision == ca.PRECISION.BF16 else quant.e4m3_table(V0)[0]
    Ue = U0.copy()
    cg = solve == ca.SOLVE_TYPE.CUMF_ALS_CG_FP32
    O.half_sweep(ptr, idx, val, Y, Ue, f, 0.05, solve=O.CG_FP32 if cg else O.CHOLESKY, cg_tol=0.0)
    if cg:  # six unconverged steps follow FP64's to the FP32 CG's tolerance
        assert rel_rows(U, Ue) < 1e-3
    else:
        assert rel_rows(U, Ue) < TOL_BF16_INPUTS
    assert not U[np.diff(ptr) == 0].any()
