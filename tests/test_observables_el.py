"""Observables of 8 and 16 bands (one thread per k point and matrix entry) and
the eigenvectors they use with a renormalised H, against the oracle at grids
whose last sub-tile, block or eigenvector group is partly filled."""
import numpy as np
import pytest

import edus_b200 as E
from edus_b200 import workloads as W
from oracle_lib import Oracle

pytestmark = pytest.mark.gpu


# 12 x 12: one sub-tile a block; 46 x 50 and 34 x 38: two a block with an odd
# count of sub-tiles, and 12 of 16 / 4 of 8 matrices in the last eigenvector block
@pytest.mark.parametrize("gauge", ["length", "velocity"])
@pytest.mark.parametrize("nw,n1,n2", [(8, 12, 12), (8, 46, 50), (16, 12, 14), (16, 34, 38)])
def test_observables_match_oracle(workdir, nw, n1, n2, gauge):
    path = W.wannier(workdir, nw=nw, nside=5, n=n1, field=0.5, photon=1.6, duration=1.0, t_fin_fs=0.1, it_res=2, name="W")
    text = open(path).read().replace(f"1 {n1} {n1}", f"1 {n1} {n2}")
    if gauge == "velocity":
        text = text.replace("Wannier\n", "Wannier\nvelocity_gauge\n")
    with open(path, "w") as f:
        f.write(text)
    p = E.parse_input(path)
    ctx = E.Context(E.Problem(p, workdir), use_graphs=False)
    ctx.step(27)
    got = ctx.obs()
    want = Oracle(p, workdir).run(27)
    assert len(got) == len(want) == 14
    for q in ("J1", "J2", "pol"):
        a, b = np.array([x[q] for x in got]), np.array([x[q] for x in want])
        # k sums of at most 2300 terms in FP64, cancelling to 1e-4 of the largest
        assert np.abs(a - b).max() <= 1e-11 * max(np.abs(b).max(), 1e-4), q
    # populations are 1 - P of filled bands, P a mean of values near 1: the bar of the other tests
    assert np.abs(np.array([x["pop"] for x in got]) - np.array([x["pop"] for x in want])).max() <= 1e-13
    for q in ("trace_dev", "p_cond_max", "p_min", "n_cond"):
        assert abs(got[-1][q] - want[-1][q]) <= 1e-12, q
