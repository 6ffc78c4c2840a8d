"""The pool that hands device buffers from one context to the next, on the CPU against fakes of the CUDA calls."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_buffer_pool(tmp_path):
    exe = str(tmp_path / "pool")
    cuda = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
    subprocess.check_call([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-pthread", "-I" + os.path.join(cuda, "include"),
                           os.path.join(HERE, "c", "buffer_pool_test.cc"), "-o", exe])
    assert subprocess.run([exe], capture_output=True, text=True).stdout == "ok\n"
