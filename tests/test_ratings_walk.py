"""The walk over a row's ratings (csrc/ratings.h) at the end of the 32-bit range, on the CPU: a handle
takes up to 2^31 - 1 ratings."""
from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def walk_exe(tmp_path_factory):
    out = tmp_path_factory.mktemp("walk") / "ratings_check"
    r = subprocess.run(["g++", "-std=c++17", "-O1",
                        f"-I{ROOT / 'cuda_als_gb300' / 'csrc'}", str(ROOT / "tests" / "cpp" / "ratings_check.cpp"),
                        "-o", str(out)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


@pytest.mark.parametrize("end", [70000, 2**31 - 1, 2**31 - 2, 2**31 - 16, 2**31 - 17, 2**31 - 129])
def test_parts_of_a_row(walk_exe, end):
    r = subprocess.run([str(walk_exe), str(end)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    assert int(r.stdout) > 0
