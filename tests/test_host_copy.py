"""Staged host copies on the host: csrc/host_copy.cpp compiled with a CUDA runtime on
host memory (tests/native/fake_cuda_copies.h), so that copies overlap as on a device."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("native") / "host_copy_check")
    csrc = os.path.join(ROOT, "gradientdomaintextureprocessing_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", csrc, "-I", os.path.join(ROOT, "tests", "native"), "-I/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "native", "host_copy_check.cpp"), os.path.join(csrc, "host_copy.cpp"),
                    "-pthread", "-o", exe], check=True)

    def run(*args):
        r = subprocess.run([exe, *args], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stdout + r.stderr
        assert r.stdout.strip().endswith("ok")
    return run


@pytest.mark.parametrize("what", ["threads", "streams"])
def test_copies_that_overlap(check, what):
    """Every copy arrives whole whatever other copies of the same object are under way."""
    check(what)


def test_systems_of_a_device_share_one(check):
    """The pinned memory and the threads do not grow with the systems and go with the last."""
    check("shared")


def test_chunks_are_made_once_they_pay(check):
    """Pinned memory costs more than the first copies gain: a program of a few calls has none."""
    check("first")


def test_threads_sleep_while_a_copy_waits(check):
    """A copy behind 0.3 s of queued work costs no processor time while it waits (five
    polling threads: 1.5 s; a copy of 12 MB itself: a few ms)."""
    check("idle")
