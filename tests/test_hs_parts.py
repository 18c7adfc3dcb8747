"""The Roering solver's block partials, on the host: each pass has a region of
its own as large as its grid (tests/hs_parts_check.cu, compiled with nvcc and
run here; it launches nothing)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_partials_do_not_overlap(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if not nvcc:
        pytest.skip("no nvcc")
    exe = str(tmp_path / "hs_parts_check")
    p = subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_103a,code=sm_103a",
                        "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "lsdtt_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "hs_parts_check.cu"), "-o", exe], capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True)
    print(r.stdout)
    assert r.returncode == 0 and r.stdout.strip().endswith("OK"), r.stdout + r.stderr
