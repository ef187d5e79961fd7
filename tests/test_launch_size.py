"""What a launch costs the host depends on the bytes of its arguments: 24 or 32
beyond a multiple of 64 are the cheap ones. The kernels that step small lattices
one launch per call take a StepConst and 72 bytes more (d = 2 strips: 80)."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "coolbubble_b200", "csrc")


def test_step_arguments_have_a_cheap_size(tmp_path):
    src, exe = tmp_path / "size.cpp", tmp_path / "size"
    src.write_text('#include <cstdio>\n#include "cb_internal.h"\nint main() { std::printf("%zu", sizeof(cb::StepConst)); }\n')
    cuda = os.environ.get("CUDA", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-I" + CSRC, "-I" + os.path.join(cuda, "include"), str(src), "-o", str(exe)],
                   check=True)
    size = int(subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout)
    assert (size + 72) % 64 in (24, 32) and (size + 80) % 64 in (24, 32), size
