"""The batched pass's plan memory (csrc/plan_memory.hpp), on the CPU against a
device of limited capacity."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_plans_in_turn(tmp_path):
    exe = tmp_path / "plan_memory_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(ROOT, "unblending_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "plan_memory_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
