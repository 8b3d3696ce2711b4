"""The math functions for arguments of a known range (an arc cosine of [0, 1],
sine and cosine of the quarter circle) equal the general ones bit for bit."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_ranged_functions_equal_the_general_ones(tmp_path):
    exe = tmp_path / "math_ranges"
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off",
                           "-I" + os.path.join(ROOT, "artemis_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "cpp", "math_ranges.cpp"), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.split() == ["0"], out.stdout + out.stderr
