"""Device buffers after an allocation that failed, on the CPU: nothing keeps what has been freed."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    out = str(tmp_path_factory.mktemp("buffers") / "eval_buffers_check")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", CUDA, "-I", os.path.join(ROOT, "ekgsim_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "native", "eval_buffers_check.cpp"), "-o", out, "-lpthread"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


@pytest.mark.parametrize("form", ["pass", "band", "dense"])
@pytest.mark.parametrize("few,many", [(1, 2), (3, 40)])
def test_buffers_after_out_of_memory(program, form, few, many):
    """A batch that does not fit ends in EKG_ERR_OUT_OF_MEMORY, and the smaller one after it gets buffers of its
    own again (the buffers of every pass, and those of the per-simulation form for both contractions)."""
    r = subprocess.run([program, form, str(few), str(many)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
