"""The passes of the spectrum that just miss the registers of one more block per SM, by what the assembler reports:
the x pass at 384 and 512 and the y pass at 320 leave room for three blocks of 256 threads, the y pass at 96 for five."""
import pathlib
import re
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
X = "template __global__ void k_green_x<{n}>(const GreenGeom, double2*, const double2*);\n"
YZ = "template __global__ void k_green_yz<{n}, 1>(const GreenGeom, const double2*, double2*, float2*, const double2*);\n"


@pytest.mark.skipif(not pathlib.Path(NVCC).exists(), reason="needs nvcc")
@pytest.mark.parametrize("kernel,n,blocks", [(X, 384, 3), (X, 512, 3), (YZ, 320, 3), (YZ, 96, 5)])
def test_blocks_per_sm(tmp_path, kernel, n, blocks):
    src = tmp_path / "g.cu"
    src.write_text('#include "green_kernels.cuh"\nnamespace ifdda {\n' + kernel.format(n=n) + "}\n")
    out = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                          "--expt-relaxed-constexpr", "-I", str(ROOT / "if-dda_b200" / "csrc"), "-I",
                          str(ROOT / "include"), "-Xptxas", "-v", "-cubin", "-o", str(tmp_path / "g.cubin"), str(src)],
                         capture_output=True, text=True, check=True).stderr
    regs = int(re.search(r"Used (\d+) registers", out).group(1))
    assert 65536 // (8 * (-(-regs * 32 // 256) * 256)) >= blocks, out  # a warp's registers come in units of 256
