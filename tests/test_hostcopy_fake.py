"""The threaded host copies against a fake CUDA runtime (tests/cpp/hostcopy_fake.cc): streams that run
nothing until they are waited for, a per-thread stream handle that names another queue in every thread, an
event that cannot be recorded, a stream in capture, owners that copy too little to pay for the threads."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "tarang_b200", "csrc")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    out = tmp_path_factory.mktemp("hostcopy") / "hostcopy_fake"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CSRC, "-I" + inc, "-x", "c++",
                    os.path.join(CSRC, "tg_hostcopy.cu"), os.path.join(HERE, "cpp", "hostcopy_fake.cc"), "-o", str(out),
                    "-lpthread"], check=True)
    return str(out)


@pytest.mark.parametrize("scenario", ["download", "upload", "download_per_thread", "upload_per_thread"])
def test_order(program, scenario):
    r = subprocess.run([program, scenario], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout


def test_no_transfer_left_in_flight(program):
    r = subprocess.run([program, "record_fails"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout


def test_stream_in_capture(program):
    r = subprocess.run([program, "capture"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout


def test_short_use_sets_up_nothing(program):
    r = subprocess.run([program, "short_use"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
