"""The line sweeps' short quotient (quick_quotient.h) against the division, on the host."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_quotients_equal_the_division(tmp_path):
    exe = str(tmp_path / "check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "code_mge_gb300", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "quick_quotient_check.cpp")], check=True)
    r = subprocess.run([exe, "4000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
