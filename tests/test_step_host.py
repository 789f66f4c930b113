"""The host side of stepping on the CPU: tests/host/step_host.cu links
fsl_group.cu with a CUDA runtime of its own that only counts, so that calls of
the runtime can be refused without a GPU."""
import os
import subprocess

import pytest

from fluam_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    exe = str(tmp_path_factory.mktemp("host") / "step_host")
    subprocess.run([nvcc] + build.ARCH + ["-std=c++17", "--expt-relaxed-constexpr", "-O0", "-cudart", "none",
                                          os.path.join(HERE, "host", "step_host.cu"), os.path.join(HERE, "host", "counting_cudart.cpp"),
                                          "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("what", ["refused", "refused_each", "io_key", "mapped"])
def test_step_host(program, what):
    r = subprocess.run([program, what], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
