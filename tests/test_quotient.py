"""The solver's division by a shared reciprocal (csrc/quotient.hpp) equals the
IEEE division it replaces on every operand tried, on the CPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_quotient_equals_division(tmp_path):
    exe = tmp_path / "quotient_check"
    subprocess.run(["g++", "-std=c++17", "-O2", "-mfma", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "unblending_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "quotient_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
