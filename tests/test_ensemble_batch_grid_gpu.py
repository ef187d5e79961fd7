"""Batch launches beyond 65535 lattices, and partial sums of as many rows as the
members have tiles (runs of that number take minutes to create: the launch is
called with members laid out by hand)."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_members_of_large_and_mixed_batches_equal_launches_of_their_own(tmp_path):
    cuda = os.environ.get("CUDA", "/usr/local/cuda")
    lib, exe = os.path.join(ROOT, "coolbubble_b200", "lib"), str(tmp_path / "batch_members")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "coolbubble_b200", "csrc"),
                    "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(cuda, "include"),
                    os.path.join(ROOT, "tests", "native", "batch_members.cpp"), "-o", exe, "-L" + lib, "-lcoolbubble_b200",
                    "-Wl,-rpath," + lib, "-L" + os.path.join(cuda, "lib64"), "-lcudart_static", "-lpthread", "-ldl", "-lrt"],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.endswith("ok\n"), r.stdout + r.stderr
