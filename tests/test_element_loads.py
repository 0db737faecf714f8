"""The loads of each element as the assembly and the gradient look them up,
without a device (element_loads_host.cpp)."""
import os
import subprocess

from yeti_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_element_loads_are_those_of_the_lists(tmp_path):
    exe = str(tmp_path / "element_loads_host")
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", build.CSRC, "-I", cuda,
                    os.path.join(HERE, "element_loads_host.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
