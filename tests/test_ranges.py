"""Overlap of buffer ranges (ranges.h), which decides how launches are ordered."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_any_overlap(tmp_path):
    exe = str(tmp_path / "ranges_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "pcg-square_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "ranges_check.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe], timeout=120).returncode == 0
