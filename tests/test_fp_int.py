"""The integer forms of FP64 comparisons, conversions, quotients and the stage
count's root (csrc/fp_int.cuh), and the device copy of the canonical math
functions, compiled for the host and compared bit for bit with FP64
arithmetic and with the oracle's copy."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "cerebellum-neuron-model-simulation-using-rkc_gb300", "csrc")
SRC = os.path.join(ROOT, "tests", "native", "fp_int_check.cpp")


def test_fp_int(tmp_path):
    exe = str(tmp_path / "fp_int_check")
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-Wall", "-ffp-contract=off", f"-I{CSRC}",
                    f"-I{os.path.join(ROOT, 'oracle')}", SRC, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip().endswith("all equal"), r.stdout + r.stderr
