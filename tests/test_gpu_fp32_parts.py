"""FP32 rows of more than 16,384 ratings, in parts, at the sizes the other test leaves out: the Gram by
patches (f <= 32, its tiles handed over through the ring) and the largest panel pitch."""
from __future__ import annotations

import pytest

import cuda_als_gb300 as ca
import test_gpu_core as core

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f", [1, 8, 9, 24, 32, 33, 129, 175, 176])
@pytest.mark.parametrize("solve", [ca.SOLVE_TYPE.CHOLESKY, ca.SOLVE_TYPE.LU])
def test_rows_in_parts(f, solve):
    core.test_fp32_rows_split_into_parts_match_the_oracle(f, solve)
