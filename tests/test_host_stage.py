"""The host-array transfers (host_stage.cpp) on the CPU: the file is compiled
against a CUDA runtime of plain host memory, with the address sanitizer where
lifetimes are checked."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pcg-square_b200", "csrc")


def build(path, *flags):
    exe = str(path / "host_stage_check")
    subprocess.run(["g++", "-std=c++17", "-g", *flags, "-I", os.path.join(ROOT, "include"), "-I", CSRC,
                    "-isystem", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "native", "host_stage_check.cpp"),
                    os.path.join(CSRC, "host_stage.cpp"), "-o", exe, "-lpthread"], check=True)
    return exe


def run(exe, *args):
    r = subprocess.run([exe, *args], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-4000:]


@pytest.fixture(scope="module")
def sanitized(tmp_path_factory):
    return build(tmp_path_factory.mktemp("asan"), "-O1", "-fsanitize=address",
                 "-fsanitize-address-use-after-scope")


# Gathered, direct, helper threads, and more than the staging buffer holds.
@pytest.mark.parametrize("mb", [1, 9, 17, 40])
def test_transfers_within_lifetimes(sanitized, mb):
    run(sanitized, "move", str(mb))


@pytest.fixture(scope="module")
def plain(tmp_path_factory):
    return build(tmp_path_factory.mktemp("plain"), "-O2")


def test_helpers_sleep_while_the_device_works(plain):
    run(plain, "idle", "16")


def test_a_thread_that_cannot_be_had(plain):
    run(plain, "threads", "17")


@pytest.mark.parametrize("mb", [3, 17])
def test_failed_transfers_leave_nothing_in_flight(sanitized, mb):
    run(sanitized, "failed", str(mb))
