"""Reads through page-locked memory (host_copy.h), compiled against a stand-in
for the CUDA runtime: what they cost the host, and what they do without memory."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "gsbn_b200", "csrc")
CHECKS = ["waiting", "chunks", "small"]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("host_copy") / "check")
    native = os.path.join(HERE, "native")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + os.path.join(native, "fake_cuda"), "-I" + CSRC,
                    os.path.join(native, "host_copy_check.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("check", CHECKS)
def test_host_copy(program, check):
    r = subprocess.run([program, check], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
