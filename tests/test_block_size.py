"""The block size asked for is the one that is launched, none asked for is the
solver's choice, and the autotuners time each size once and report what ran:
the host code of the single-phase solver and the pool on a CUDA runtime of
host memory (cpp/block_size.cpp).  Built with g++ here; no GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "jianhui-lbm_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")),
                    reason="needs g++ and the CUDA headers")
def test_block_sizes(tmp_path):
    exe = tmp_path / "block_size"
    srcs = [os.path.join(CSRC, s) for s in ("batch.cpp", "api.cpp", "transfer.cpp", "geometry.cpp", "mrt.cpp")]
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", os.path.join(CUDA, "include"), "-I",
                    os.path.join(ROOT, "include"), "-I", CSRC, *srcs, os.path.join(ROOT, "tests", "cpp", "block_size.cpp"),
                    "-no-pie", "-rdynamic", "-Wl,--unresolved-symbols=ignore-all", "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
