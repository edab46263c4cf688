"""Registers of the kernels of single solves, as the compiler reports them: the blocks
per SM that each band count is sized for, and no more spills than there were."""
import os
import re
import subprocess

import pytest

from edus_b200 import build as B


def report(source, pattern, tmp):
    """Groups of `pattern` (the kernel's mangled name), spill bytes and registers of every match."""
    flags = [f for f in B.NVCC_FLAGS if f != "-lineinfo"]
    r = subprocess.run([B.nvcc(), "-c", os.path.join(B.CSRC, "cuda", source), "-o", str(tmp / "k.o"), "-Xptxas", "-v"] + flags,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    found = re.finditer(r"Compiling entry function '\S*" + pattern + r".*?(\d+) bytes spill stores.*?Used (\d+) registers", r.stderr, re.S)
    return [tuple(int(x) for x in m.groups()) for m in found]


@pytest.fixture(scope="module")
def rhs(tmp_path_factory):
    out = {}
    for n, kt, dyn, spill, regs in report("rhs_ep.cu", r"k_rhs_epILi(\d+)ELi(\d+)ELb(\d)E", tmp_path_factory.mktemp("rhs")):
        warps = (kt * n * (n + 1) // 2 + 31) // 32
        out[n, bool(dyn)] = dict(spill=spill, blocks=65536 // ((regs + 7) // 8 * 8 * 32 * warps))
    return out


@pytest.mark.parametrize("n,dyn,blocks,spill", [
    (1, False, 18, 0), (2, False, 7, 0), (3, False, 4, 0), (4, False, 2, 0), (5, False, 1, 0), (8, False, 3, 100), (16, False, 1, 148),
    (1, True, 18, 0), (2, True, 7, 8), (3, True, 4, 32), (4, True, 1, 0), (5, True, 1, 0),
])
def test_resident_blocks(rhs, n, dyn, blocks, spill):
    assert rhs[n, dyn]["blocks"] >= blocks and rhs[n, dyn]["spill"] <= spill, rhs[n, dyn]


def test_observables_spill_no_more_than_the_products_need(tmp_path):
    spill = {n: b for n, b, _ in report("obs.cu", r"k_obsILi(\d+)E", tmp_path)}
    assert spill[3] == 0 and spill[5] <= 1776
