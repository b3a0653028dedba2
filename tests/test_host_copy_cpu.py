"""The threaded copies between pageable host memory and the device
(csrc/host_copy.h), linked with a CUDA runtime of the test's own whose streams
run as late as the ordering rules allow: what the copies rely on is then seen
every time and without a GPU."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CUDA_INCLUDE = Path("/usr/local/cuda/include")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx or not (CUDA_INCLUDE / "cuda_runtime_api.h").exists():
        pytest.skip("no g++ or CUDA headers")
    exe = tmp_path_factory.mktemp("host_copy") / "check"
    subprocess.run([gxx, "-std=c++17", "-O1", "-pthread", "-I", str(CUDA_INCLUDE), "-I", str(ROOT / "iroiro_b200/csrc"),
                    str(ROOT / "tests/host_copy_check.cpp"), "-o", str(exe)], check=True)
    return exe


@pytest.mark.parametrize("what", ["other_context", "route", "no_pinned_memory", "per_thread_stream"])
def test_host_copy(check, what):
    """other_context: an upload on one context's stream, with DMAs still
    queued, then copies of another context of the same device.
    route: the sizes from which a copy goes through the slots, by direction and
    by whether the destination was touched before.
    no_pinned_memory: the allocation of the slots fails; the copies go on.
    per_thread_stream: a context on cudaStreamPerThread."""
    r = subprocess.run([str(check), what], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
