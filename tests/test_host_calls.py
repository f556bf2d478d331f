"""The library's host code on a fake CUDA runtime (tests/cuda/host_check.cpp: no GPU):
what calls keep between them, and what they share."""
import os
import subprocess

import pytest

from gpu_optical_photons_b200 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def host_check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("host") / "host_check")
    src = [os.path.join(HERE, "cuda", f) for f in ("host_check.cpp", "fake_cudart.cpp")]
    subprocess.run([B.nvcc()] + B.ARCH + ["-O1", "-std=c++17", "-cudart", "none", "-x", "cu", "-I", B.CSRC,
                                          "-I", B.INCLUDE]
                   + src + [os.path.join(B.CSRC, "capi.cu"), "-o", exe, "-lpthread", "-ldl"], check=True)
    return exe


@pytest.mark.parametrize("check", ["devices", "overlap", "graphs", "kept", "sizes", "threads", "forked", "stale",
                                   "wide_blocks", "routes"])
def test_host_code(host_check, check):
    out = subprocess.run([host_check, check], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
