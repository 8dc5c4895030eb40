"""Host vectors copied to the device (DBuf::upload_vec in internal.hpp) may be
temporaries: the layout builds hand over vectors that end with the statement or
the block. Run against a stand-in for the CUDA runtime whose asynchronous
copies read their source only when the stream is waited for."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "helm-project_gb300", "csrc")
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.mark.parametrize("n,empty_first", [(1, 0), (5, 1), (100000, 0), (3, 1)])
def test_vector_may_go_after_the_call(tmp_path, n, empty_first):
    gxx = shutil.which("g++")
    if gxx is None or not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers not available")
    out = str(tmp_path / "libupload.so")
    subprocess.run([gxx, "-std=c++20", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", CSRC, "-I", CUDA,
                    os.path.join(HERE, "native", "upload_harness.cpp"), "-o", out], check=True)
    assert C.CDLL(out).uploaded(n, empty_first) == n
