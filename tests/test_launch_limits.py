"""A kernel's shared-memory limit serves every launch of it, whatever sizes other
threads and other plans use it for. Without a GPU: the launch code linked to a
stand-in for the CUDA runtime (host_runtime/fake_launch.cpp) that refuses what the
runtime refuses."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "high-order-regularization_b200")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def _program(d, cpp, cu, more=()):
    """The program of host_runtime/*.cpp sources and the package's .cu files."""
    objs = []
    for f in cu:
        objs.append(str(d / (f + ".o")))
        subprocess.run([os.environ.get("NVCC", os.path.join(CUDA, "bin", "nvcc")), "-gencode", "arch=compute_100a,code=sm_100a",
                        "-std=c++17", "--expt-relaxed-constexpr", "-c", os.path.join(PKG, "csrc", f), "-o", objs[-1]], check=True)
    exe = str(d / "program")
    subprocess.run(["g++", "-O1", "-g", "-std=c++17", "-fopenmp", "-I", os.path.join(CUDA, "include"),
                    *(os.path.join(HERE, "host_runtime", f) for f in cpp), *more, *objs, "-o", exe], check=True)
    return exe


def _run(exe, *args):
    r = subprocess.run([exe, *args], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def test_upward_passes_of_two_degrees(tmp_path):
    _run(_program(tmp_path, ["upward_cases.cpp", "fake_launch.cpp"], ["hr_aux.cu", "hr_moments_tc.cu"]))


def test_sine_transform_plans_of_two_sizes(tmp_path):
    _run(_program(tmp_path, ["dst_cases.cpp", "fake_cudart.cpp", "fake_launch.cpp"], ["hr_poisson.cu", "hr_runtime.cu"],
                  [os.path.join(PKG, "host", "hr_tree.cpp")]))
