"""The transforms' lazy signed arithmetic on the CPU, under the signed-overflow
sanitizer: 2p is only 2^28 below 2^63, so the order of an addition matters."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_signed_ranges(tmp_path):
    exe = str(tmp_path / "ntt_range_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=undefined",
                    "-fno-sanitize-recover=undefined", "-x", "c++",
                    "-I", os.path.join(ROOT, "pcg-square_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "ntt_range_check.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
