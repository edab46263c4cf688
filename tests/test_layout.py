"""States and tables between the reference's layout and the device's planes: a
last block that is partly filled, every band count, the staged copy's last piece."""
import numpy as np
import pytest

import edus_b200 as E
from edus_b200 import abi
from edus_b200 import workloads as W

pytestmark = pytest.mark.gpu


# 4 x 4: less than a block of 32 k points; 10 x 12: 24 in the last; 130 x 130 with 8
# bands: 17.3 MB, four full pinned buffers and a ragged piece
@pytest.mark.parametrize("nw,n", [(2, 4), (3, 10), (5, 10), (8, 12), (16, 6), (8, 130)])
def test_batch_state_before_the_first_step(workdir, nw, n):
    if nw == 3:
        path = W.hbn_rk4(workdir, n=n, t_fin_fs=0.1)
    else:
        path = W.wannier(workdir, nw=nw, nside=3, n=n, t_fin_fs=0.1, name="W")
    pb = E.Problem(E.parse_input(path), workdir)
    rho0 = pb.get("P0")
    b = E.Batch(precision=abi.EDUS_PREC_FP64)
    s = b.add(pb)
    assert np.array_equal(b.get_state(s), _hermitian(rho0))
    c = E.Context(pb)
    assert np.array_equal(c.get_state(), _hermitian(rho0))
    if nw >= 4:
        m = E.Batch(precision=abi.EDUS_PREC_MIXED)
        assert np.array_equal(m.get_state(m.add(pb)), _hermitian(rho0))  # deviation 0 + rho_eq


def _hermitian(a):
    """the device keeps the upper triangle"""
    up = np.triu(a)
    return up + np.conj(np.triu(a, 1)).transpose(0, 2, 1)
