"""Device memory is given back when a construction ends with an error, on the CPU: the owners of mw_internal.hpp with a counting
allocator that can fail (tests/cpp/scratch.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_memory_is_given_back_after_errors(tmp_path):
    exe = str(tmp_path / "scratch")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "mrchem_b200", "csrc"),
                           "-I" + os.path.join(CUDA, "include"), os.path.join(ROOT, "tests", "cpp", "scratch.cpp"), "-o", exe])
    lines = subprocess.check_output([exe], text=True).split("\n")[:-1]
    # name, whether it ended with an error, arrays still held
    assert lines == ["scratch 0 0", "scratch 1 0", "scratch 1 0", "scratch 1 0", "tables 0 0", "tables 1 0", "duplicate 0 0", "kept 0 1"]
