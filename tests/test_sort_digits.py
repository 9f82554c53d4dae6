"""The radix sort's choice of digits (octree_gb300/csrc/otg_radix.h) keeps the order of the keys."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_digits_order_keys(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ missing")
    exe = str(tmp_path / "sort_digits")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(HERE, "..", "octree_gb300", "csrc"),
                    os.path.join(HERE, "cpp", "sort_digits_test.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe], capture_output=True, text=True, check=True).stdout.strip() == "ok"
