"""The projection's tiles divide a cell's divergence by its number of fluid
neighbours, 0 to 4, as the product by the number's reciprocal. That must give the
bits of the reference's fast-math division (apply_projection_at,
src/fluid.cu:240) for every input: compared over all 2^32 float bit patterns on
the GPU."""
import os
import subprocess

import pytest

from tests.conftest import ROOT

SRC = ROOT / "tests" / "cpp" / "count_division.cu"
EXE = ROOT / "oracle" / "build" / "count_division"


def build_program():
    if EXE.exists() and SRC.stat().st_mtime <= EXE.stat().st_mtime:
        return EXE
    EXE.parent.mkdir(parents=True, exist_ok=True)
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    cmd = [nvcc, "-std=c++17", "-O3", "--use_fast_math", "-gencode",
           "arch=compute_103a,code=sm_103a", str(SRC), "-o", str(EXE)]
    subprocess.run(cmd, check=True, capture_output=True, text=True)
    return EXE


def test_program_compiles():
    assert build_program().exists()


@pytest.mark.gpu
def test_products_equal_divisions_by_every_count(gpu):
    out = subprocess.run([str(build_program())], check=True, capture_output=True, text=True,
                         timeout=120).stdout.strip().splitlines()
    assert len(out) == 5
    assert not [line for line in out if line.split()[1] != "0"], out
