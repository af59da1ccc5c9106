"""A field read that runs out of device memory and is made again: the host code
of the two-phase, solute and pool solvers on a CUDA runtime of host memory
(cpp/field_read_retry.cpp), every allocation of a read failed in turn.  Built
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
    out = tmp_path_factory.mktemp("retry") / "field_read_retry"
    srcs = [os.path.join(CSRC, s) for s in ("cg_api.cpp", "st7_api.cpp", "batch.cpp", "api.cpp", "transfer.cpp",
                                            "geometry.cpp", "mrt.cpp")]
    # the launchers no field read reaches stay undefined
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", os.path.join(CUDA, "include"), "-I",
                    os.path.join(ROOT, "include"), "-I", CSRC, *srcs,
                    os.path.join(ROOT, "tests", "cpp", "field_read_retry.cpp"),
                    "-no-pie", "-rdynamic", "-Wl,--unresolved-symbols=ignore-all", "-o", str(out)], check=True)
    return str(out)


@pytest.mark.parametrize("args", [[], ["nopin"]])
def test_read_after_out_of_memory(exe, args):
    """nopin: no host memory can be pinned, as under a limit on locked memory;
    the handles are created and read all the same."""
    r = subprocess.run([exe, *args], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
