"""The rule that lets a marching kernel use one set of row-end offsets for both
vectors of a thread, against the offsets themselves (host arithmetic)."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "coolbubble_b200", "csrc")

SOURCE = r"""
#include <cstdio>
#include "cb_internal.h"
int main() {
    int taken = 0;
    for (int prec = 0; prec < 2; ++prec)
        for (int n = 64; n <= 1024; ++n)
            for (int t = 2; t <= 40 && t <= n; ++t) {
                const int W = prec == 0 ? 2 : 4, nv = n / W;
                if (!cb::whole_rows(n, cb::run_pitch(3, n, prec), prec, t)) continue;
                ++taken;
                /* as the kernels place them: vectors u and u + threads of the tile, threads in whole warps */
                const int threads = (t * nv + 63) / 64 * 32;
                if (2 * threads != t * nv || n % t != 0) return std::printf("threads: %d %d %d\n", prec, n, t), 1;
                for (int u = 0; u < threads; ++u) {
                    const int a = W * u % n, b = W * (u + threads) % n;
                    if (a != b) return std::printf("sites: %d %d %d at %d\n", prec, n, t, u), 1;
                    if (u % 32 == 0 && a + 32 * W > n) return std::printf("warps: %d %d %d at %d\n", prec, n, t, u), 1;
                }
            }
    std::printf("%d\n", taken);
    return taken < 100;
}
"""


def test_both_vectors_of_a_thread_start_at_the_same_site(tmp_path):
    src, exe = tmp_path / "whole.cpp", tmp_path / "whole"
    src.write_text(SOURCE)
    cuda = os.environ.get("CUDA", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CSRC, "-I" + os.path.join(cuda, "include"), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
