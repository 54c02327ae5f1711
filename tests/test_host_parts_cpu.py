"""Parts of the library that a host compiler can run without a device
(tests/cpp): the stage kernel's ring protocol on host threads, with waits that run
out in some lanes only; the table of kernels that may be launched; the staged
copies of the host-buffer operator over a fake runtime; the list of restricted cells."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CXX = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"


def build(out, name):
    cpp = os.path.join(ROOT, "tests", "cpp")
    subprocess.run([CXX, "-std=c++17", "-O1", "-pthread", "-ldl", "-I", os.path.join(cpp, "host_cuda"),
                    "-I", os.path.join(ROOT, "granite_b200", "csrc"), os.path.join(cpp, name + ".cpp"),
                    "-o", str(out / name)], check=True)
    return str(out / name)


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    return build(tmp_path_factory.mktemp("ring"), "test_stage_ring")


@pytest.mark.parametrize("what", ["tiles", "selected", "load_lane_late 0", "load_lane_late 9", "compute_lane_late 0",
                                  "compute_lane_late 13",
                                  # the run has 154 items: one in its midst, and those before the end of the list
                                  "compute_warps_late 28", "compute_warps_late 151", "compute_warps_late 153"])
def test_ring(exe, what):
    r = subprocess.run([exe, *what.split()], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip() == "OK"


def test_every_kernel_answers_for_its_registers(tmp_path):
    r = subprocess.run([build(tmp_path, "test_tma_grids")], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("what", ["staged", "no_pinned", "no_events", "no_threads", "no_thread_state", "copy_error",
                                  "capture_elsewhere"])
def test_host_copies(tmp_path, what):
    r = subprocess.run([build(tmp_path, "test_host_copy"), what], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


def test_restriction_list(tmp_path):
    r = subprocess.run([build(tmp_path, "test_restrict_list")], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
