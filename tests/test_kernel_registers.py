"""Resident CTAs that a kernel's timing rests on, from the register counts that
ptxas prints (no GPU): with 73 registers or more the binning kernel's 128-thread
CTAs fit an SM six times instead of seven, which cost the binning stage 12 %
of 3M Gaussians once when a refactoring raised the count."""
from __future__ import annotations

import re
import subprocess
from pathlib import Path

import pytest

from gamesplat_b200 import build as B

SM_REGISTERS, WARP_GRANULE = 65536, 256   # an SM's file; a warp's registers come in such pieces


def _registers(source: str, kernel: str, out: Path) -> int:
    try:
        cc = B.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")
    r = subprocess.run([cc, *B.ARCH, "-lineinfo", "-std=c++17", "-O3", "-I", str(B.PKG.parent / "include"), "-Xptxas",
                        "-v", "-c", str(B.CSRC / source), "-o", str(out)], capture_output=True, text=True, check=True)
    blocks = re.split(r"Compiling entry function '", r.stdout + r.stderr)[1:]
    counts = [int(re.search(r"Used (\d+) registers", b).group(1)) for b in blocks if kernel in b.split("'")[0]]
    assert len(counts) == 1, (kernel, len(counts))
    return counts[0]


@pytest.mark.parametrize("source,kernel,threads,ctas", [("gs_bin.cu", "10bin_kernel", 128, 7)])
def test_resident_ctas(source, kernel, threads, ctas, tmp_path):
    regs = _registers(source, kernel, tmp_path / "k.o")
    warp = -(-regs * 32 // WARP_GRANULE) * WARP_GRANULE
    assert SM_REGISTERS // (warp * threads // 32) >= ctas, regs
