"""The ensemble's one-kernel stage refuses a term count that no kernel was built for, before any CUDA call."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_term_counts_without_a_kernel_are_refused(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path / "ens_stage_terms")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O1", "-std=c++17", "-o", exe,
                    os.path.join(HERE, "native", "ens_stage_terms.cu")], check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "refused 4 of 4\n", r.stdout + r.stderr
