"""Registers of the stage kernel of single solves, as the compiler reports them: the
blocks per SM that each band count is sized for, and no spills where there were none."""
import os
import re
import subprocess

import pytest

from edus_b200 import build as B


@pytest.fixture(scope="module")
def rhs(tmp_path_factory):
    src = os.path.join(B.CSRC, "cuda", "rhs_ep.cu")
    flags = [f for f in B.NVCC_FLAGS if f != "-lineinfo"]
    r = subprocess.run([B.nvcc(), "-c", src, "-o", str(tmp_path_factory.mktemp("o") / "rhs.o"), "-Xptxas", "-v"] + flags, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = {}
    for m in re.finditer(r"k_rhs_epILi(\d+)ELi(\d+)ELb(\d)E.*?(\d+) bytes spill stores.*?Used (\d+) registers", r.stderr, re.S):
        n, kt, dyn, spill, regs = (int(x) for x in m.groups())
        threads = kt * n * (n + 1) // 2
        warps = (threads + 31) // 32
        out[n, bool(dyn)] = dict(spill=spill, blocks=65536 // ((regs + 7) // 8 * 8 * 32 * warps))
    return out


@pytest.mark.parametrize("n,dyn,blocks,spill", [
    (1, False, 18, 0), (2, False, 7, 0), (3, False, 4, 0), (4, False, 2, 0), (5, False, 1, 0), (8, False, 3, 100), (16, False, 1, 148),
    (1, True, 18, 0), (2, True, 7, 8), (3, True, 4, 32), (4, True, 1, 0), (5, True, 1, 0),
])
def test_resident_blocks(rhs, n, dyn, blocks, spill):
    assert rhs[n, dyn]["blocks"] >= blocks and rhs[n, dyn]["spill"] <= spill, rhs[n, dyn]
