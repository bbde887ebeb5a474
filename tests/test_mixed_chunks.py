"""The mixed tile kernel's source chunks (csrc/plan_tools.h), compiled alone on the CPU."""
import os
import re
import subprocess

NATIVE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")


def test_chunk_counts(tmp_path):
    """The time of a chunking against its CTAs dealt out one by one; the count taken is within 15 % of the
    best by it, and the sizes that lost by six tiles a chunk take others."""
    exe = str(tmp_path / "mixed_chunks_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", exe, os.path.join(NATIVE, "mixed_chunks_check.cpp")], check=True,
                   capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    cases, bad = map(int, re.search(r"cases (\d+) bad (\d+)", r.stdout).groups())
    assert cases > 10000 and bad == 0
