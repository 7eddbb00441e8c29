"""Sizes of the operator lists (mw_opplan.hpp), on the CPU: records are counted in 64 bits, a group whose lists are large is
built one operator at a time, and one operator's lists beyond 32-bit positions are refused."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("plan") / "op_plan")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "mrchem_b200", "csrc"),
                           os.path.join(ROOT, "tests", "cpp", "op_plan.cpp"), "-o", exe])
    return lambda nop, rows, scan, records: subprocess.check_output([exe] + [str(v) for v in (nop, rows, scan, records)], text=True).strip()


def sizes(nop, nterm, boxes):
    """rows, scanned offsets and records at the root, where every offset of a term whose band is the world's width is listed"""
    w = 2 * (boxes - 1) + 1
    return nop, nop * nterm * w ** 2, nop * nterm * w ** 3, nop * nterm * w ** 3


@pytest.mark.parametrize("nop,nterm,boxes,want", [
    (8, 134, 10, "together"),  # the standard world
    (1, 134, 40, "together"),
    (8, 100, 70, "singly"),    # 2,148,495,200 records: more than a 32-bit count holds
    (2, 134, 4, "together"),
    (1, 30, 256, "refuse"),    # 4e9 records of one operator
    (8, 30, 256, "singly"),    # each of them is then refused by itself
])
def test_plan_of_wide_roots(plan, nop, nterm, boxes, want):
    assert plan(*sizes(nop, nterm, boxes)) == want


def test_plan_edges(plan):
    assert plan(8, 1000, 1e9, 2 ** 24) == "together" and plan(8, 1000, 1e9, 2 ** 24 + 1) == "singly"
    assert plan(1, 1000, 1e9, 2 ** 31 - 1024) == "together" and plan(1, 1000, 1e9, 2 ** 31 - 1023) == "refuse"
    assert plan(1, 2 ** 30, 1e9, 5) == "together" and plan(1, 2 ** 30 + 1, 1e9, 5) == "refuse"
    assert plan(2, 2 ** 24 + 1, 1e9, 5) == "singly"
    assert plan(1, 2 ** 24, 1e11, 5) == "together" and plan(1, 2 ** 24, 1.01e11, 5) == "refuse"
    assert plan(2, 2 ** 24, 1.01e11, 5) == "singly"
