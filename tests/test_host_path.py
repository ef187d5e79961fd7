"""The library's host code on a fake of the CUDA runtime (no GPU): downloads that
fail half-way or find little room, and what a run's first steps launch."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "coolbubble_b200", "csrc")


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fake") / "fake_cuda")
    cuda = os.environ.get("CUDA", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(cuda, "include"), os.path.join(ROOT, "tests", "native", "fake_cuda.cpp"),
                    os.path.join(CSRC, "cb_api.cpp"), os.path.join(CSRC, "cb_pool.cpp"), "-x", "c++",
                    os.path.join(CSRC, "cb_ensemble.cu"), "-o", exe, "-lpthread"], check=True)
    return exe


def run(exe, what):
    r = subprocess.run([exe, what], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr


def test_a_failed_download_leaves_no_copy_under_way(fake):
    run(fake, "download")


def test_a_served_run_without_its_fields_hands_out_zeros(fake):
    run(fake, "served")


def test_first_steps_launch_their_steps_and_wait_for_nothing(fake):
    run(fake, "first")


def test_padded_fields_come_down_where_the_device_has_little_room(fake):
    run(fake, "room")


def test_an_ensemble_reports_a_member_whose_wait_ran_out(fake):
    run(fake, "ensemble")
