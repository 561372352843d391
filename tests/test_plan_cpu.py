"""CPU check of the rules that choose a call's kernel mode and a range's pieces (csrc/kv_plan.h, host code)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def build(tmp_path):
    exe = str(tmp_path / "plan_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "qwen38-megakernel_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "plan_check.cpp")], check=True)
    return exe


def test_mode_and_pieces_depend_on_the_bucket_only(tmp_path):
    r = subprocess.run([build(tmp_path)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
