"""Batch observables of 8 and 16 bands at grids whose last unit and last run of k
points are partly filled, against the single solve of the same problem."""
import numpy as np
import pytest

import edus_b200 as E
from edus_b200 import abi
from edus_b200 import workloads as W

pytestmark = pytest.mark.gpu


# 4 x 4: less than one unit; 12 x 14 = 128 + 40 k points, 40 = 2 x 16 + 8; 10 x 14 = 2 x 64 + 12
@pytest.mark.parametrize("nw,n1,n2", [(8, 4, 4), (8, 12, 14), (16, 4, 4), (16, 10, 14)])
@pytest.mark.parametrize("prec", [abi.EDUS_PREC_FP64, abi.EDUS_PREC_MIXED])
def test_batch_observables_match_single_solve(workdir, nw, n1, n2, prec):
    path = W.wannier(workdir, nw=nw, nside=5, n=n1, field=0.5, photon=1.6, duration=0.8, t_fin_fs=0.3, it_res=5, name="W")
    text = open(path).read().replace(f"1 {n1} {n1}\n", f"1 {n1} {n2}\n")
    with open(path, "w") as f:
        f.write(text)
    pb = E.Problem(E.parse_input(path), workdir)
    ctx = E.Context(pb)
    ctx.run()
    b = E.Batch(precision=prec)
    s = b.add(pb)
    while b.poll(s)[0] != abi.EDUS_INST_DONE:
        b.advance(16)
    got, want = b.obs(s), ctx.obs()
    assert len(got) == len(want)
    # FP64: k sums in another order; mixed: the tables and the stage inputs are FP32
    # (6e-8 each, some 50 steps), sums of at most 168 x 256 terms of order one
    tol = 1e-12 if prec == abi.EDUS_PREC_FP64 else 2e-5
    for q in ("J1", "J2", "pol", "pop", "trace_dev", "p_cond_max", "p_min", "n_cond"):
        x, y = np.array([o[q] for o in got]), np.array([o[q] for o in want])
        assert np.abs(x - y).max() <= tol * max(1.0, np.abs(y).max()), q
