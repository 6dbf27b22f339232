"""The DIC/DILU sweeps keep a chunk of slots in registers (kernels.cuh:
SweepShape): no form of them may spill, since a spilled chunk goes back and
forth through local memory at every poll.  Compiled here for the GPU, no
device needed; the figures are the assembler's own report."""
import os
import re
import shutil
import subprocess

import pytest

from programs_b200.build import CSRC, NVCC_FLAGS, _nvcc

SOURCE = "#include \"kernels.cuh\"\n" + "".join(
    f"template __global__ void sg::k_{d}_sf<{t}, {v}, {g}>("
    f"int, sg::Rows<{t}>, sg::SweepMap, const {t}*, const {t}*, {t}*, {t}*, sg::SweepCtl*, "
    "const int*);\n"
    for d in ("fwd", "bwd") for t in ("double", "float") for v in (1, 2, 3, 4)
    for g in ("true", "false"))


@pytest.mark.skipif(shutil.which("c++filt") is None, reason="needs binutils")
def test_no_sweep_spills(tmp_path):
    src = tmp_path / "sweeps.cu"
    src.write_text(SOURCE)
    flags = [f for f in NVCC_FLAGS if f not in ("-shared", "-lineinfo")]
    r = subprocess.run([_nvcc(), *flags, "-I", CSRC, "-Xptxas", "-v", "-c", str(src), "-o",
                        os.path.join(tmp_path, "sweeps.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run(["c++filt"], input=r.stderr, capture_output=True, text=True).stdout
    seen = re.findall(r"Compiling entry function '(?:void )?(sg::k_(?:fwd|bwd)_sf<.*?>).*?"
                      r"(\d+) bytes spill stores, (\d+) bytes spill loads", out, re.S)
    assert len(seen) == 32
    assert [x for x in seen if x[1] != "0" or x[2] != "0"] == []
