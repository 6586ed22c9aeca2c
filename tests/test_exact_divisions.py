"""The division-free quotients of the block quantiser (csrc/gv_exact.h) equal IEEE division, the tanh GELU by table the function."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_quotients_equal_ieee_division(tmp_path):
    probe = tmp_path / "probe"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma", "-o", str(probe),
                    os.path.join(ROOT, "tests", "exact_divisions_probe.cpp")], check=True)
    assert subprocess.run([str(probe)], check=True, capture_output=True, text=True).stdout.strip() == "0"
