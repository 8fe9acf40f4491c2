"""zconv's register caps, by what the assembler reports: the shapes whose middle has five points (z lengths 10, 20 and
40) keep their values in registers in FP64, and spill at most 32 bytes a thread in FP32."""
import pathlib
import re
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not pathlib.Path(NVCC).exists(), reason="needs nvcc")
@pytest.mark.parametrize("real,limit", [("double", 0), ("float", 32)])
def test_five_point_middles_stay_in_registers(tmp_path, real, limit):
    lengths = (10, 20, 40)
    src = tmp_path / "z.cu"
    src.write_text('#include "matvec_kernels.cuh"\nnamespace ifdda {\n' + "".join(
        f"template __global__ void k_zconv<{real}, {n}, MvTiles<{real}, {n}, 0>>(const MvArgs<{real}>);\n"
        for n in lengths) + "}\n")
    out = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                          "--expt-relaxed-constexpr", "-I", str(ROOT / "if-dda_b200" / "csrc"), "-I",
                          str(ROOT / "include"), "-Xptxas", "-v", "-cubin", "-o", str(tmp_path / "z.cubin"), str(src)],
                         capture_output=True, text=True, check=True).stderr
    spills = [int(n) for n in re.findall(r"(\d+) bytes spill stores", out)]
    assert len(spills) == len(lengths) and max(spills) <= limit, out
