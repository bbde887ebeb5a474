"""The event screens of the certified FP64 form leave inactive bodies out: one merged body, parked at
1e20 AU, would widen the Hill screen over every pair."""
import os
import re
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_screen_maxima_leave_inactive_bodies_out(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "cert_screen_gpu")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-fmad=false", "-o", exe,
                    os.path.join(HERE, "native", "cert_screen_gpu.cu")], check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert re.search(r"systems 5 bad 0", r.stdout)
