"""Handle buffers (csrc/memory.cu) over a fake CUDA runtime that refuses calls
(tests/cpp/memory_fake_runtime.cpp): no GPU needed."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("memory") / "memory_fake_runtime")
    csrc = os.path.join(ROOT, "spc5_b200", "csrc")
    cmd = ["g++", "-std=c++17", "-I", csrc, "-I", os.path.join(ROOT, "include"), "-I", "/usr/local/cuda/include",
           os.path.join(ROOT, "tests", "cpp", "memory_fake_runtime.cpp"), "-x", "c++", os.path.join(csrc, "memory.cu"),
           "-o", exe]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-3000:]

    def run(scenario):
        res = subprocess.run([exe, scenario], capture_output=True, text=True, timeout=60)
        assert res.returncode == 0, (scenario, res.returncode, res.stderr)  # < 0: std::terminate
        return res.stdout.split("\n")[:-1]

    return run


def test_a_buffer_goes_back_after_the_device_wait(fake):
    assert fake("plain") == ["cudaMalloc", "cudaFree", "cudaFreeAsync", "mode as before", "last error 0", "done"]


def test_the_wait_happens_beside_a_capture(fake):
    """Beside a capture in the global mode the wait is made in the relaxed mode,
    and the thread's mode is put back."""
    assert fake("capture") == ["cudaMalloc", "cudaFree", "cudaFreeAsync", "mode as before", "last error 0", "done"]


def test_a_buffer_is_kept_when_the_wait_is_refused(fake):
    """Memory that some stream may still use does not go back to the pool, and
    the refusals are not left for the next call to report."""
    assert fake("no_wait") == ["cudaMalloc refused", "cudaDeviceSynchronize refused", "mode as before", "last error 0",
                               "done"]


def test_a_release_does_not_throw(fake):
    """While the runtime unloads, a destructor has nothing to give back and must
    not end the process."""
    assert fake("unloading") == ["cudaGetDevice refused", "mode as before", "last error 0", "done"]
