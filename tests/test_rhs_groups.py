"""Stage kernel of single solves: the selected stencil vectors are taken in groups, the
first two by themselves, the rest in a loop. Vector counts below, at and past the ends of the
groups for every band count, against the oracle; the adaptive step's kernel against the
same loop driven by the host."""
import numpy as np
import pytest

import edus_b200 as E
from edus_b200 import abi
from edus_b200 import workloads as W
from oracle_lib import Oracle

pytestmark = pytest.mark.gpu


def write(workdir, model, n, extra=""):
    if isinstance(model, int):
        path = W.wannier(workdir, nw=model, nside=3, n=n, name="W", t_fin_fs=0.4, duration=0.4, it_res=5)
    else:
        path = W.hbn_rk4(workdir, n=n, t_fin_fs=0.4, duration=0.4, field=0.5, photon=1.6, it_res=5)
    text = open(path).read().replace("tdse{\n", "tdse{\n" + extra)
    if not isinstance(model, int):
        lines = text.splitlines()
        q = next(i for i, x in enumerate(lines) if x.startswith("tightbinding"))
        text = "\n".join(lines[:q] + ["tightbinding " + model] + lines[q + 1:]) + "\n"
    with open(path, "w") as f:
        f.write(text)
    return path


HBN = "Haldane_CoreBN_Nedge gap= 5.8 t1= 2.3 t2= 0 phi0= 0"


# vectors with a coefficient: 14 and 18 (2 bands), 10 and 12 (hexagonal, 3 and 4 bands), 8 and
# 12, of which 4 and 8 are left (square: 5 and 8 bands); 1 band: a square stencil too
@pytest.mark.parametrize("model,n", [("BN1b", 6), ("Vampa2015", 10), (HBN, 6), ("Graphene_costD", 10), (5, 6), (8, 6), (16, 6)])
@pytest.mark.parametrize("field", [(0.0, 0.0, 0.0), (0.0, 4e-4, 0.0), (0.0, 0.0, -3e-4), (0.0, 3e-4, 2e-4)])
def test_derivative_matches_oracle(workdir, model, n, field):
    p = E.parse_input(write(workdir, model, n))
    pb = E.Problem(p, workdir)
    ctx, o = E.Context(pb), Oracle(p, workdir)
    rng = np.random.default_rng(3)
    P = pb.get("P0")
    X = (rng.standard_normal(P.shape) + 1j * rng.standard_normal(P.shape)) * 0.01
    P = P + X + np.conj(np.transpose(X, (0, 2, 1)))
    EF = list(field) + [0.0, 0.0, 0.0]
    ctx.slot_set(abi.SLOT_P0, P)
    ctx.get_derivative(abi.SLOT_P0, EF, p.probe.wl, int(any(field)))
    g = ctx.slot_get(abi.SLOT_PV)
    r = o.rhs(P, EF, p.probe.wl, int(any(field)))
    # sums of up to 18 gradient terms w E b P of about 1e2 x 4e-4 x P each, and n products
    assert np.abs(g - r).max() <= 1e-14 * max(1.0, np.abs(r).max() * 10)


@pytest.mark.parametrize("model,n", [("BN1b", 6), ("Vampa2015", 10), (HBN, 6), ("Graphene_costD", 10), (5, 6), (8, 6)])
def test_adaptive_run_matches_the_host_loop(workdir, model, n, monkeypatch):
    pb = E.Problem(E.parse_input(write(workdir, model, n, "dynamical_dt_evolution\nepsStepAbs 0.001\n")), workdir)
    a, b = E.Context(pb), E.Context(pb)
    a.run()
    monkeypatch.setenv("EDUS_DYN_HOST", "1")
    b.run()
    assert a.clock()[0] == b.clock()[0]
    assert np.abs(a.get_state() - b.get_state()).max() < 1e-10  # the step size carries the rounding of a small change


# the terms that are left out are zero for finite states only: 0 x inf is not
@pytest.mark.parametrize("model,n", [("Vampa2015", 10), (HBN, 6), (8, 6)])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1e300])
def test_state_that_is_not_finite_reaches_every_neighbour(workdir, model, n, value):
    p = E.parse_input(write(workdir, model, n))
    pb = E.Problem(p, workdir)
    ctx, o = E.Context(pb), Oracle(p, workdir)
    P = pb.get("P0")
    P[n + 1, 0, 1] = complex(0.0, value)
    P[n + 1, 1, 0] = complex(0.0, -value)
    EF = [0.0, 0.0, 4e-4, 0.0, 0.0, 0.0]
    ctx.slot_set(abi.SLOT_P0, P)
    ctx.get_derivative(abi.SLOT_P0, EF, p.probe.wl, 1)
    g, r = ctx.slot_get(abi.SLOT_PV), o.rhs(P, EF, p.probe.wl, 1)
    upper = np.triu(np.ones(P.shape[1:], bool))
    assert np.array_equal(np.isfinite(g)[:, upper], np.isfinite(r)[:, upper])
    assert np.isfinite(value) == np.isfinite(g).all()
