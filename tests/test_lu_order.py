"""The row order that the one-launch band LU's blocks take from a panel's pivots:
it must not depend on anything that block 0 writes again in later panels, since a
block may lag by any number of them."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_row_order_from_pivots(tmp_path):
    exe = str(tmp_path / "lu_order")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(ROOT, "piro_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "lu_order.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0
