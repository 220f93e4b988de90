"""Addresses of the robust normalisation's wavefront (sigpde_b200/csrc/norm_wave.cuh), walked on the host."""
import os
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_norm_wave_addresses_stay_in_their_regions(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "norm_bounds_check"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--expt-relaxed-constexpr", "-I",
                    os.path.join(ROOT, "sigpde_b200", "csrc"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "norm_bounds_check.cu")], check=True, capture_output=True, timeout=600)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
