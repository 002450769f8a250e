"""The device memory of shape sets, on the CPU: the library's own objects linked against a stand-in for
the CUDA runtime (tests/cpp/fake_cudart.cpp) that keeps a log of the calls and a limit on the memory."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
OBJ = os.path.join(ROOT, "curvami-official_gb300", "_build")
CPP = os.path.join(ROOT, "tests", "cpp")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    import __graft_entry__ as ge

    ge.build()
    exe = str(tmp_path_factory.mktemp("memory") / "shape_memory")
    cuda = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", os.path.join(cuda, "include"),
                           os.path.join(CPP, "shape_memory.cpp"), os.path.join(CPP, "fake_cudart.cpp")]
                          + [os.path.join(OBJ, u + ".o") for u in ("shape", "pattern", "assemble", "capi", "noalloc", "batch")]
                          + ["-o", exe])
    return exe


@pytest.mark.parametrize("what", ["failed_set", "destroy", "room", "scratch", "trim"])
def test_memory(program, what):
    r = subprocess.run([program, what], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
