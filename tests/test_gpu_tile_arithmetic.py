"""The reciprocals and quotients of the register-tile solvers against CUDA's division, and the solvers
against the column-at-a-time ones: bit for bit over their range of pivots, and by their errors against
FP64 beyond (tests/cpp/tile_check.cu)."""
from __future__ import annotations

import subprocess

import pytest

from cuda_als_gb300 import build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tile_exe(tmp_path_factory):
    src = build.PKG.parent / "tests" / "cpp" / "tile_check.cu"
    out = tmp_path_factory.mktemp("tile") / "tile_check"
    r = subprocess.run([build.nvcc(), "-std=c++17", "-O3", f"-I{build.CSRC}", str(src), *build.ARCH,
                        "-o", str(out)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


@pytest.mark.parametrize("what", ["reciprocal", "quotients", "solve"])
def test_the_tiles_arithmetic_to_the_bit(tile_exe, what):
    r = subprocess.run([str(tile_exe), what], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    rows = [line.split() for line in r.stdout.splitlines()]
    assert rows and all(int(n) > 0 for _, n, _ in rows)
    assert [(name, bad) for name, _, bad in rows if int(bad)] == []
