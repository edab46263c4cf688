"""Child processes that run the product's library over a stand-in CUDA runtime
(fake_cudart.c): what the host code does when a call of the runtime fails, and
which kernels it launches, without a GPU."""
import os
import subprocess
import sys
import textwrap

from conftest import ROOT

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PRELUDE = """
import ctypes as C, os, sys
sys.path.insert(0, {root!r})
import numpy as np
import edus_b200 as E
from edus_b200 import abi, workloads as W
F = C.CDLL("libcudart.so.12")
F.fake_launches.restype = F.fake_graph_launches.restype = C.c_long
F.fake_held.restype = C.c_size_t
F.fake_set.argtypes = [C.c_char_p, C.c_long]
def limit(name, v): assert F.fake_set(name.encode(), v) == 0
def launches(part=""): return F.fake_launches(part.encode())
def problem(path, **kw): return E.Problem(E.parse_input(path), os.path.dirname(path), **kw)
d = {work!r}
"""


def run_host(work, body, **env):
    """Run `body` after PRELUDE in a child whose libcudart is the stand-in."""
    libs = os.path.join(work, "runtime")
    os.makedirs(libs, exist_ok=True)
    so, ver = os.path.join(libs, "libcudart.so.12"), os.path.join(libs, "version.map")
    with open(ver, "w") as f:
        f.write("libcudart.so.12 { global: *; };\n")
    subprocess.run(["gcc", "-std=gnu11", "-shared", "-fPIC", "-O1", "-I" + os.path.join(CUDA, "include"), os.path.join(HERE, "fake_cudart.c"),
                    "-o", so, "-Wl,-soname,libcudart.so.12", "-Wl,--version-script=" + ver], check=True)
    e = dict(os.environ, LD_LIBRARY_PATH=libs + ":" + os.environ.get("LD_LIBRARY_PATH", ""), **env)
    r = subprocess.run([sys.executable, "-c", PRELUDE.format(root=ROOT, work=work) + textwrap.dedent(body)], capture_output=True, text=True,
                       env=e, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return r.stdout
