"""csrc/fp_int.cuh on the GPU, against the GPU's own FP64 divide, conversions,
comparisons and square root (tests/native/fp_int_gpu.cu): 200 million random
pairs, none of which may differ.  (A quotient lies within the correction's
error of a midpoint for one pair in 2^51, so this expects 2e-7 of them.)"""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "cerebellum-neuron-model-simulation-using-rkc_gb300", "csrc")
SRC = os.path.join(ROOT, "tests", "native", "fp_int_gpu.cu")


def _nvcc():
    return os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")


def _compile(out):
    subprocess.run([_nvcc(), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-fmad=false", f"-I{CSRC}",
                    SRC, "-o", out], check=True)


def test_compiles(tmp_path):
    _compile(str(tmp_path / "fp_int_gpu"))


@pytest.mark.gpu
def test_fp_int_on_the_gpu(tmp_path):
    exe = str(tmp_path / "fp_int_gpu")
    _compile(exe)
    r = subprocess.run([exe, "200"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("all equal"), r.stdout + r.stderr
