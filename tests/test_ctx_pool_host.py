"""The context's allocations without a device: ctx.cu compiled against a CUDA
runtime that keeps lists (ctx_pool_host.cpp)."""
import os
import subprocess

import pytest

from yeti_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("ctx_pool") / "ctx_pool_host")
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    subprocess.run(["g++", "-std=c++17", "-I", build.CSRC, "-I", os.path.join(build.ROOT, "include"),
                    "-I", cuda, os.path.join(HERE, "ctx_pool_host.cpp"),
                    "-x", "c++", os.path.join(build.CSRC, "ctx.cu"), "-pthread", "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("scenario", ["sizes", "device_just_large_enough", "budget", "reuse", "given_back",
                                      "order"])
def test_pool(harness, scenario):
    r = subprocess.run([harness, scenario], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
