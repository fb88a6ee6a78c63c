"""Which epochs are replayed from CUDA graphs: the calls of cudaGraphLaunch are counted in a program
linked from the library's objects."""
from __future__ import annotations

import subprocess

import pytest

import cuda_als_gb300 as ca
from cuda_als_gb300 import build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph_exe(tmp_path_factory):
    src = build.PKG.parent / "tests" / "cpp" / "graph_main.cpp"
    out = tmp_path_factory.mktemp("graph") / "graph_main"
    objs = [str(build.OBJDIR / (s.replace(".", "_") + ".o")) for s in build.SOURCES]
    r = subprocess.run([build.nvcc(), "-std=c++17", "-O1", f"-I{build.INCLUDE}", str(src), *objs, *build.ARCH,
                        "-Xcompiler", "-fopenmp", "-lgomp", "-Xlinker", "--wrap=cudaGraphLaunch",
                        "-o", str(out)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


def _run(exe, precision, solve, use_graph, calls):
    r = subprocess.run([str(exe), str(int(precision)), str(int(solve)), str(use_graph), *map(str, calls)],
                       capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    *rows, same = r.stdout.split("\n")[:-1]
    assert same == "equal"
    rows = [tuple(map(int, row.split())) for row in rows]
    assert all(timed for _, timed in rows)  # every call measures its last half-sweeps
    return [n for n, _ in rows]


@pytest.mark.parametrize("precision,solve", [
    (ca.PRECISION.FP32, ca.SOLVE_TYPE.LU), (ca.PRECISION.BF16, ca.SOLVE_TYPE.CHOLESKY),
    (ca.PRECISION.FP8, ca.SOLVE_TYPE.CUMF_ALS_CG_FP32)])
def test_every_epoch_after_the_first_is_replayed(graph_exe, precision, solve):
    """One epoch a call, as a program that evaluates in between does, and several: a graph or more an
    epoch once one has run eagerly."""
    for calls, eager in (([1, 1, 1, 3], 1), ([4], 1), ([2], 1)):
        launches = _run(graph_exe, precision, solve, 1, calls)
        for n, epochs in zip(launches, calls):
            assert n == 0 if epochs == eager else n >= epochs - eager
            eager = 0
    assert _run(graph_exe, precision, solve, 0, [1, 1, 3]) == [0, 0, 0]
