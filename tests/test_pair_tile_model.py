"""CPU: the index arithmetic of the pair tiles (two transforms per thread) is walked
element by element for every tile shape of a range of lengths: bounds of the
shared-memory words, every butterfly once, and the transform itself; and the rounding
of the inter-pass twiddles."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("nvcc") is None and not os.path.exists("/usr/local/cuda/bin/nvcc"),
                    reason="nvcc not available")
def test_pair_tile_indices(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "pair_check"
    src = os.path.join(ROOT, "tests", "host", "pair_check.cu")
    subprocess.check_call([nvcc, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-Wno-deprecated-gpu-targets",
                           "-I", os.path.join(ROOT, "sip_b200", "csrc"), "-o", str(exe), src])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "ALL OK" in r.stdout
