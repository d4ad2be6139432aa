"""The library's host code under a stand-in CUDA runtime (fake_cudart.cpp): the order of uploads and kernels, what
error returns leave behind, and memory budgets.  No GPU; each check runs in a process of its own (host_calls.py)."""

import os
import re
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CHECKS = re.findall(r"^def check_(\w+)", open(os.path.join(HERE, "host_calls.py")).read(), re.M)


@pytest.fixture(scope="session")
def fake(tmp_path_factory, native_lib):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    out = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-std=c++17", "-I", inc, os.path.join(HERE, "fake_cudart.cpp"),
                    "-o", out], check=True)
    return out


@pytest.mark.parametrize("check", CHECKS)
def test_host_calls(fake, check):
    p = subprocess.run([sys.executable, os.path.join(HERE, "host_calls.py"), fake, check], capture_output=True,
                       text=True, env={**os.environ, "LD_PRELOAD": fake}, timeout=300)
    assert p.returncode == 0, p.stdout + p.stderr
