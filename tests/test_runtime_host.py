"""Host logic of the runtime (csrc/hr_runtime.h, .cu) without a GPU: compiled
as C++ against a stand-in for the CUDA runtime (host_runtime/)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "high-order-regularization_b200")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def cases(tmp_path_factory):
    d = tmp_path_factory.mktemp("host_runtime")
    src = [os.path.join(HERE, "host_runtime", "cases.cpp"), os.path.join(HERE, "host_runtime", "fake_cudart.cpp"),
           os.path.join(PKG, "host", "hr_tree.cpp")]
    exe = str(d / "cases")
    subprocess.run(["g++", "-O1", "-g", "-std=c++17", "-fopenmp", "-I", os.path.join(CUDA, "include"), *src, "-x", "c++",
                    os.path.join(PKG, "csrc", "hr_runtime.cu"), "-o", exe], check=True)
    return exe


def _run(cases, name):
    r = subprocess.run([cases, name], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("name", ["failed_growth", "page_locked_copies", "no_page_locked_memory", "workspace_growth", "workspace_given_back", "order_of_items"])
def test_case(cases, name):
    _run(cases, name)
