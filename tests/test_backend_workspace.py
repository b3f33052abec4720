"""Scratch buffers of the host mirrors, on the CPU: what a captured graph was recorded with has to stay."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_cpp_mirror(tmp_path):
    """The C++ mirror over fakes of the CUDA runtime and the library (tests/cpp/workspace_tests.cpp)."""
    from aidotnet.tensors_b200 import build
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc())))
    exe = str(tmp_path / "workspace_tests")
    # the entry points that no case reaches have no fake
    subprocess.run([build._host_cxx(), "-std=c++17", "-O1", "-g", "-I", os.path.join(cuda, "include"), "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "workspace_tests.cpp"),
                    os.path.join(build.CSRC, "host", "direct_gpu_backend.cpp"), "-Wl,--unresolved-symbols=ignore-in-object-files"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "all cases passed" in r.stdout, r.stdout + r.stderr
