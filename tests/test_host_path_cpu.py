"""CPU: the host-array path (host_path.cu, memory.cu) against a model of the CUDA runtime, in a process of its own
(tests/host_path_harness.cc): what it does between threads and when a call of the runtime fails."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "tetris-artifact-evalution_b200", "csrc")


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not os.path.exists(os.path.join(include, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    exe = str(tmp_path_factory.mktemp("harness") / "harness")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-pthread", "-I", include, "-x", "c++", os.path.join(CSRC, "memory.cu"),
                    os.path.join(CSRC, "host_path.cu"), os.path.join(ROOT, "tests", "host_path_harness.cc"), "-o", exe], check=True)
    return exe


def _run(harness, scenario):
    res = subprocess.run([harness, scenario], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stderr


def test_release_waits_for_a_call_that_uses_the_copy_streams(harness):
    _run(harness, "release_race")


@pytest.mark.parametrize("scenario", ["upload_error", "download_error", "upload_mark_error"])
def test_an_error_of_the_device_ends_a_staged_copy(harness, scenario):
    _run(harness, scenario)


def test_staged_copies_take_no_memory(harness):
    _run(harness, "no_memory")


@pytest.mark.parametrize("scenario", ["idle_helpers", "helper_budget"])
def test_helpers_take_no_cores_they_do_not_use(harness, scenario):
    _run(harness, scenario)


def test_an_upload_does_not_wait_for_another_streams(harness):
    _run(harness, "busy_ring")


def test_a_slot_at_work_does_not_hold_back_idle_slots(harness):
    _run(harness, "slot_in_use")
