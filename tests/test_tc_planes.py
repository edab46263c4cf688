"""The tensor-core contraction that forms its slice pairs itself, at the edges of its
tiles: the planes of the cp.async-staged form, bit for bit (every FP32 sum of either is
exact, so nothing but the layout can differ)."""
import numpy as np
import pytest

import edus_b200 as E
from edus_b200 import abi
from edus_b200 import workloads as W

pytestmark = pytest.mark.gpu


# R vectors nside^2: one chunk (9), a full group (121), part of a second group (169), two full
# groups (225), part of a third (289); columns 8 nw (nw + 1) / 2: 24 and 48 (part of a tile),
# 120 (a tile and a half), 288, 1088; k points n^2: part of a tile, 128 + 16, two full tiles
@pytest.mark.parametrize("nw,nside,n", [(2, 3, 10), (2, 17, 12), (3, 13, 12), (5, 11, 16), (5, 15, 10), (8, 15, 12), (16, 11, 12)])
def test_planes_form_equals_cp_async_form(workdir, monkeypatch, nw, nside, n):
    path = W.wannier(workdir, nw=nw, nside=nside, n=n, name="W", field=0.5, t_fin_fs=0.1, it_res=5)
    text = open(path).read()
    results = []
    for form in ("", "cpasync"):
        monkeypatch.setenv("EDUS_TC_GEMM", form)
        with open(path, "w") as f:
            f.write(text.replace("Wannier\n", "Wannier\nvelocity_gauge\n"))
        ctx = E.Context(E.Problem(E.parse_input(path), workdir), precision=abi.EDUS_PREC_MIXED)
        ctx.run()
        with open(path, "w") as f:
            f.write(text)
        b = E.Batch(precision=abi.EDUS_PREC_MIXED, tc_contraction=True)
        s = b.add(E.Problem(E.parse_input(path), workdir, defer_model=True))
        while b.poll(s)[0] != abi.EDUS_INST_DONE:
            b.advance(16)
        results.append((ctx.get_state(), np.array([o["J1"] for o in ctx.obs()]), b.get_state(s), np.array([o["J1"] for o in b.obs(s)])))
    for x, y in zip(*results):
        assert np.array_equal(x, y)
        assert np.isfinite(x).all()
