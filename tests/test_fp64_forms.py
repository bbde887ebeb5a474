"""The FP64 plan's rules (csrc/plan_tools.h), compiled alone on the CPU."""
import os
import re
import subprocess

NATIVE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")


def test_block_forms_and_pair_parallel_sinks(tmp_path):
    """fp64_block_form on both sides of each line and along a block's sinks; PairparSinks against waves
    and steps counted one by one."""
    exe = str(tmp_path / "fp64_forms_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", exe, os.path.join(NATIVE, "fp64_forms_check.cpp")], check=True,
                   capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    cases, bad = map(int, re.search(r"cases (\d+) bad (\d+)", r.stdout).groups())
    assert cases > 200000 and bad == 0
