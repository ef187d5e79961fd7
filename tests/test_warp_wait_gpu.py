"""The bounded waits of the staged kernels give one answer per warp."""
import ctypes
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "coolbubble_b200", "csrc")
NVCC = os.path.join(os.environ.get("CUDA", "/usr/local/cuda"), "bin", "nvcc")


def test_a_wait_that_runs_out_in_some_lanes_has_run_out_in_all(tmp_path):
    """Lanes 0..15 give up at once, lanes 16..31 would wait until the phase
    completes: the warp's answer is no, in every lane (the kernels' shuffles
    follow under it). Once the phase has completed the answer is yes, in every
    lane."""
    so = str(tmp_path / "warp_wait.so")
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-I" + CSRC, os.path.join(HERE, "native", "warp_wait.cu"), "-o", so], check=True)
    out = (ctypes.c_int * 64)()
    assert ctypes.CDLL(so).run_warp_wait(out) == 0
    assert list(out[:32]) == [0] * 32
    assert list(out[32:]) == [1] * 32
