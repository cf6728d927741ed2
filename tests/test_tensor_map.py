"""The lookup of the driver's tensor map encoder, by threads that make their first searches at the same time."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_first_searches_of_several_threads(tmp_path):
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if not os.path.exists(os.path.join(cuda, "cuda.h")):
        pytest.skip("no CUDA headers")
    exe = str(tmp_path / "tensor_map_test")
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", cuda, "-I", os.path.join(ROOT, "faiss-metal_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "tensor_map_test.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], stdout=subprocess.PIPE, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
