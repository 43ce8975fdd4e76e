"""The single-row bulk-copy GEMV keeps up to six groups a lane (K <= 6144) in registers: what ptxas reports for it, by the compiler that
builds the library."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dgx-serving_b200", "csrc")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def test_bulk_copy_gemv_does_not_spill(tmp_path):
    if not shutil.which(NVCC):
        pytest.skip("no nvcc")
    src = tmp_path / "bulk.cu"
    src.write_text('#include "common.cuh"\n#include "peer_allgather.cuh"\n#include "gemv_w4a8_bulk.cuh"\n')
    out = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xptxas", "-v", "-c", "-I", CSRC, "-o",
                          str(tmp_path / "bulk.o"), str(src)], check=True, capture_output=True, text=True)
    report = re.findall(r"Function properties for \S*gemv_w4a8_bulk_kernelILi(\d)E(f|6__half)Lb0ELb0E\S*\n.*?(\d+) bytes spill stores", out.stdout + out.stderr)
    spills = {(int(groups), scales): int(n) for groups, scales, n in report}
    assert len(spills) == 16 and all(spills[g, s] == 0 for g in range(1, 7) for s in ("f", "6__half")), spills
