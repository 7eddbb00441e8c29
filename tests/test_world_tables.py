"""A failed allocation while a world's first operator is made leaves the world without operator tables, not with half of them, and
its next operator makes them (on the CPU, tests/cpp/world_tables.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_failed_first_operator(tmp_path):
    exe = str(tmp_path / "world_tables")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "mrchem_b200", "csrc"),
                           "-I" + os.path.join(CUDA, "include"), os.path.join(ROOT, "tests", "cpp", "world_tables.cpp"), "-o", exe])
    # failed, has tables, has all of them after the next call; allocation 0, 1, 2 fails, then none
    assert subprocess.check_output([exe], text=True).split("\n")[:-1] == ["1 0 1", "1 0 1", "1 0 1", "0 1 1"]
