"""The clustering's labels (csrc/ec.cu label_kernel) do not rest on every node
hanging directly under its root: tests/native/ec_label_check.cu."""
import pathlib
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = tmp_path_factory.mktemp("ec") / "ec_label_check"
    csrc = ROOT / "daphne-benchmark_b200" / "csrc"
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "--fmad=false", "-Xcompiler", "-fopenmp", "-I", str(csrc), "-o", str(exe),
                    str(ROOT / "tests" / "native" / "ec_label_check.cu"), str(csrc / "grid_build.cu"),
                    str(csrc / "ec_pose.cpp")], check=True)
    return exe


@pytest.mark.parametrize("n", [4, 33, 256, 1000, 40000])
def test_labels_of_deep_trees(program, n):
    r = subprocess.run([str(program), str(n)], capture_output=True, text=True, check=True)
    assert r.stdout.strip() == "0"
