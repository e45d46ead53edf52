"""Registers of the GEMM instances that carry a fused push (the kernels of several ranks): 20 and 16 warps share the register file, so a
change to code that all instances share can push values of the tile loop into local memory.  The compiler's own report, no GPU."""
import os
import re
import shutil
import subprocess

import pytest

from streamep_b200 import _ext

NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no CUDA compiler")
@pytest.mark.parametrize("source,name", [("gemm_inst_swiglu.cu", "A"), ("gemm_inst_dswiglu.cu", "Y_bwd")])
def test_spills_of_fused_push_instances(source, name, tmp_path):
    out = subprocess.run([NVCC, *_ext.NVCC_FLAGS, "-Xptxas", "-v", "-cubin", "-o", str(tmp_path / "x.cubin"), str(_ext._CSRC / source)],
                         capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr[-2000:]
    report = re.findall(r"Compiling entry function '(\w*grouped_gemm_kernel\w*)'.*?(\d+) bytes spill stores, (\d+) bytes spill loads", out.stderr, re.S)
    # template arguments <tile width, A and B MN-major, epilogue, push, CTAs of a unit>
    push = {m: (int(stores), int(loads)) for m, stores, loads in report if re.search(r"ILi\d+ELb\dELb\dELi\dELb1ELi\dE", m)}
    assert len(push) == 3 and len(report) == 6, out.stderr[-2000:]
    for instance, (stores, loads) in push.items():
        assert stores <= 12 and loads <= 12, (name, instance, stores, loads)     # bytes a thread: three registers
    assert all(int(s) == 0 and int(ld) == 0 for m, s, ld in report if m not in push)
