"""How many steps of a call are launched one by one and how many chains are
captured, for calls of every length: the host code of the single-phase and
solute solvers on a CUDA runtime of host memory (cpp/step_chains.cpp).  Built
with g++ here; no GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "jianhui-lbm_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    out = tmp_path_factory.mktemp("chains") / "step_chains"
    srcs = [os.path.join(CSRC, s) for s in ("st7_api.cpp", "api.cpp", "transfer.cpp", "geometry.cpp", "mrt.cpp")]
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", os.path.join(CUDA, "include"), "-I",
                    os.path.join(ROOT, "include"), "-I", CSRC, *srcs, os.path.join(ROOT, "tests", "cpp", "step_chains.cpp"),
                    "-no-pie", "-rdynamic", "-Wl,--unresolved-symbols=ignore-all", "-o", str(out)], check=True)
    return str(out)


@pytest.mark.parametrize("solver", ["flow", "solute"])
def test_steps_and_chains_of_a_call(exe, solver):
    r = subprocess.run([exe, solver], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
