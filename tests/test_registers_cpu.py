"""Register allocation of wavefront kernels that have few registers to spare (nvcc's own report, no GPU)."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "sigpde_b200", "csrc")


@pytest.mark.parametrize("header,kernel,params", [
    # two Gram entries of 16 coarse rows a lane: long paths of one or two dimensions
    ("stream.cuh", "stream_reg_dual_kernel<16, 0, 2, 32>", "StreamParams")])
def test_no_spills(tmp_path, header, kernel, params):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src = tmp_path / "one.cu"
    src.write_text(f'#include "{header}"\nnamespace sigk {{ template __global__ void {kernel}({params}); }}\n')
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                        "--expt-relaxed-constexpr", "-I", CSRC, "-Xptxas", "-v", "-c", str(src), "-o",
                        str(tmp_path / "one.o")], check=True, capture_output=True, text=True, timeout=600)
    spills = re.findall(r"(\d+) bytes spill stores, (\d+) bytes spill loads", r.stderr)
    assert spills and all(s == ("0", "0") for s in spills), r.stderr
