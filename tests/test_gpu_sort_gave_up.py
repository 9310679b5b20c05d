"""A wait of the radix sort that gives up (csrc/chain.cuh) ends the sort
without a write out of place and without segments (tests/native/sort_gave_up.cu:
one, two and three passes, small and large tiles)."""
import pathlib
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = tmp_path_factory.mktemp("sort") / "sort_gave_up"
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "--fmad=false", "-I", str(ROOT / "daphne-benchmark_b200" / "csrc"), "-o", str(exe),
                    str(ROOT / "tests" / "native" / "sort_gave_up.cu")], check=True)
    return exe


@pytest.mark.parametrize("n", [4097, 100000, 600001])
@pytest.mark.parametrize("bits", [7, 13, 22])
def test_sort_that_gave_up(program, n, bits):
    r = subprocess.run([str(program), str(n), str(bits)], capture_output=True, text=True)
    assert r.stdout.strip() == "ok", r.stdout + r.stderr
