"""Operator tables are built once, from the look for them to their insertion, whichever threads ask (on the CPU,
tests/cpp/op_require.cpp: eight threads, three operators, four depths)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_each_table_is_built_once(tmp_path):
    exe = str(tmp_path / "op_require")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", "-I" + os.path.join(ROOT, "mrchem_b200", "csrc"),
                           "-I" + os.path.join(CUDA, "include"), os.path.join(ROOT, "tests", "cpp", "op_require.cpp"), "-o", exe])
    for _ in range(3):
        assert subprocess.check_output([exe], text=True).split() == ["12", "0"]
