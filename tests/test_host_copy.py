"""The staging threads of the host entries, on a system that refuses threads or memory, and while there is nothing to copy.

``host_copy_check.cpp`` compiles ``csrc/host_copy.h`` against a stand-in for the CUDA runtime."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    from rustorch_b200 import build
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc())))
    exe = str(tmp_path_factory.mktemp("host_copy") / "check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-rdynamic", "-isystem", os.path.join(cuda, "include"), "-o", exe,
                    os.path.join(HERE, "host_copy_check.cpp"), "-ldl"], check=True, capture_output=True, text=True)
    return exe


@pytest.mark.parametrize("what", ["threads", "memory", "idle"])
def test_staging(program, what):
    r = subprocess.run([program, what], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.endswith("ok\n"), (r.returncode, r.stdout, r.stderr)
