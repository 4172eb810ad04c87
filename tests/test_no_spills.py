"""Kernels written to fit their registers: ptxas reports no spills for them."""
import os
import re
import subprocess

import pytest

from raster_b200 import build


@pytest.mark.parametrize("source,kernel", [("attn.cu", "gqa_decode"), ("dx.cu", "dx_tmem_kernel"), ("gemm_tc.cu", "gemm_tmem_kernel")])
def test_kernel_does_not_spill(tmp_path, source, kernel):
    try:
        nvcc = build._nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    r = subprocess.run([nvcc, *build.NVCC_FLAGS, "-Xptxas", "-v", "-c", os.path.join(build.CSRC, source), "-o", str(tmp_path / "x.o"),
                        "-I", os.path.join(build.HERE, "..", "include")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    said = re.findall(r"Compiling entry function '(\w+)'.*?(\d+) bytes spill stores", r.stderr, re.S)
    mine = [(n, int(b)) for n, b in said if kernel in n]
    assert mine and not [n for n, b in mine if b], mine
