"""The denoiser's device allocations under memory pressure, against a fake CUDA
runtime (tests/native/denoiser_alloc_check.cpp)."""
import os
import subprocess

import pytest

from nostrum_pray_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "nostrum_pray_gb300", "csrc")
OUT_OF_MEMORY = "2"


@pytest.fixture(scope="session")
def alloc_check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("alloc") / "alloc_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", os.path.join(build.CUDA_HOME, "include"), "-o", exe,
                    os.path.join(ROOT, "tests", "native", "denoiser_alloc_check.cpp"),
                    os.path.join(CSRC, "denoise_net.cpp")], check=True)

    def run(*args):
        r = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=60)
        assert r.returncode == 0, (r.returncode, r.stderr)
        return r.stdout.split()

    return run


@pytest.mark.parametrize("tensor_cores", [1, 0])
@pytest.mark.parametrize("left", [0, 1 << 20, 5 << 20])
def test_failed_backward_gives_its_buffers_back(alloc_check, tensor_cores, left):
    """A backward pass that finds no memory leaves nothing allocated behind, so
    that a retry starts where the first try did; with memory it succeeds."""
    forward, *tries = alloc_check("backward", tensor_cores, left)
    codes, used = zip(*(t.split(":") for t in tries))
    assert codes == (OUT_OF_MEMORY,) * 3 + ("0",)
    assert used[:3] == (forward,) * 3
    assert int(used[3]) > int(forward)


def test_failed_resize_fails_again(alloc_check):
    """A pass of another size that finds no memory is not taken for a made one
    by the next call of that size, which would run without buffers."""
    assert alloc_check("resize") == ["0", OUT_OF_MEMORY, OUT_OF_MEMORY, "0"]
