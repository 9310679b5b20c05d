"""The step kernel's 6x6 solve by one warp (csrc/warp_solve.cuh) gives the bits
of the serial solve: general, symmetric, zero-column, dependent-row, equal-
pivot, non-finite and zero systems (tests/native/solve_check.cu)."""
import pathlib
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = tmp_path_factory.mktemp("solve") / "solve_check"
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "--fmad=false", "-I", str(ROOT / "daphne-benchmark_b200" / "csrc"), "-o", str(exe),
                    str(ROOT / "tests" / "native" / "solve_check.cu")], check=True)
    return exe


@pytest.mark.parametrize("kind", range(7))
def test_warp_solve_bits(program, kind):
    r = subprocess.run([str(program), str(kind)], capture_output=True, text=True, check=True)
    assert r.stdout.strip() == "0"
