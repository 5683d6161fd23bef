"""Calls that only a C++ program can make (tests/host_calls.cu): populations refused after an exception, and device
populations whose sources are the list's own columns."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    from flamegpu2_gb300.build import ARCH, CORE_LIB, CUDA_HOME, LIBDIR, NVCC
    assert os.path.exists(CORE_LIB)
    exe = str(tmp_path_factory.mktemp("host_calls") / "host_calls")
    subprocess.run([NVCC] + ARCH + ["-std=c++20", "--expt-relaxed-constexpr", "-cudart", "shared",
                                    "-I", os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "host_calls.cu"),
                                    "-o", exe, "-L" + LIBDIR, "-lflamegpu2_gb300", "-Xlinker", "-rpath", "-Xlinker", LIBDIR,
                                    "-Xlinker", "-rpath", "-Xlinker", os.path.join(CUDA_HOME, "lib64")], check=True)
    return exe


@pytest.mark.parametrize("which", ["unset_id", "own_columns"])
def test_host_calls(program, which):
    r = subprocess.run([program, which], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
