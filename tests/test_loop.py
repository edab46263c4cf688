"""Whole constant-dt solves in one launch (k_loop) against the launch per stage on
the same problem, at the sizes where the split over blocks can go wrong: a
block that is partly filled, one cluster and many blocks, the largest grids the
form takes and the first it leaves to the launch per stage, every band count it
is built for, several launches in a row."""
import threading

import numpy as np
import pytest

import edus_b200 as E
from edus_b200 import abi
from edus_b200 import workloads as W
from conftest import GOLDEN_INPUT

pytestmark = pytest.mark.gpu


def make(workdir, kind, n1, n2, solver, res, t_fin=0.35):
    kw = dict(n=n1, field=0.5, photon=1.6, duration=0.8, t_fin_fs=t_fin, it_res=res)
    if kind == "hbn":
        path = W.hbn_rk4(workdir, solver=solver, **kw)
    else:
        path = W.wannier(workdir, nw=kind, nside=5, name="W", pol="0 1 1", **kw)
    text = open(path).read().replace(f"1 {n1} {n1}\n", f"1 {n1} {n2}\n")
    with open(path, "w") as f:
        f.write(text)
    return E.Problem(E.parse_input(path), workdir)


AB4 = "Adams_Bashforth 4\nAdams_Bashforth_RK4_startup\n"


@pytest.mark.parametrize("kind,n1,n2,solver,one", [
    ("hbn", 4, 4, "", True),       # one block of 16 k points
    ("hbn", 30, 32, "", True),     # 960 = 15 x 64 k points: the largest cluster
    ("hbn", 30, 34, "", True),     # the first grid past it
    ("hbn", 60, 62, AB4, True),    # last block partly filled
    ("hbn", 98, 98, "", True),     # more than kLoopSmall threads a block
    ("hbn", 98, 98, AB4, True),
    ("hbn", 118, 122, AB4, True),
    (5, 66, 66, AB4, True),
    ("hbn", 124, 124, "", True),   # 105 k points a block, the last that fits
    ("hbn", 126, 126, "", False),  # launch per stage
    (2, 12, 14, "", True),
    (4, 12, 14, "", True),
    (5, 20, 22, "", True),
    (5, 80, 80, "", False),
])
def test_one_launch_matches_launch_per_stage(workdir, kind, n1, n2, solver, one):
    pb = make(workdir, kind, n1, n2, solver, 3)
    a, b = E.Context(pb), E.Context(pb, use_graphs=False)
    for _ in range(2):  # a second run after a reset
        a.run()
        assert (a.last_timing()[1] == 1) == one
        b.run()
        # the stage arithmetic is the same expression by expression: the repository's bar for rho
        assert np.abs(a.get_state() - b.get_state()).max() <= 1e-13
        la, lb = a.obs(), b.obs()
        assert len(la) == len(lb)
        for q in ("t", "J1", "J2", "pol", "pop", "EF_pump", "trace_dev", "p_cond_max", "p_min", "n_cond", "dt"):
            x, y = np.array([o[q] for o in la]), np.array([o[q] for o in lb])
            # k sums in another order: FP64 rounding of sums whose terms are at most a few a.u.
            assert np.abs(x - y).max() <= 1e-12, q
        assert a.clock() == b.clock()
        a.reset()
        b.reset()


# stage inputs through distributed shared memory (one cluster): one block, two, a last block
# that is partly filled, all 15
@pytest.mark.parametrize("kind,n1,n2,solver", [("hbn", 4, 4, AB4), ("hbn", 6, 6, ""), ("hbn", 18, 22, AB4), ("hbn", 30, 32, AB4), (2, 24, 26, ""), (5, 18, 20, AB4)])
def test_one_cluster_matches_launch_per_stage(workdir, kind, n1, n2, solver):
    test_one_launch_matches_launch_per_stage(workdir, kind, n1, n2, solver, True)


def compare(pb):
    """One launch against the launch per stage: state, every field of the records."""
    a, b = E.Context(pb), E.Context(pb, use_graphs=False)
    a.run()
    assert a.last_timing()[1] == 1
    b.run()
    assert np.abs(a.get_state() - b.get_state()).max() <= 1e-13
    la, lb = a.obs(), b.obs()
    assert len(la) == len(lb) > 2
    for q in la[0]:
        x, y = np.array([o[q] for o in la]), np.array([o[q] for o in lb])
        assert np.abs(x - y).max() <= 1e-12, q
    return lb


# a decaying core hole (relaxation), circular pump, probe on the core, transient absorption:
# one cluster, many blocks, blocks of more than kLoopSmall threads
@pytest.mark.parametrize("n1,n2", [(12, 14), (40, 40), (100, 100)])
@pytest.mark.parametrize("solver", ["Adams_Bashforth 5", ""])
def test_core_hole_in_one_launch(workdir, n1, n2, solver):
    text = open(GOLDEN_INPUT).read().replace("1 70 70", f"1 {n1} {n2}").replace("Adams_Bashforth\n", solver + "\n")
    text = "\n".join(x for x in text.splitlines() if not x.startswith("PrintPopulation")) + "\n"
    text = text.replace("t_fin 1650.36549334624544 au", "t_fin 92.0 au")  # the probe follows the pump
    with open(workdir + "/input.txt", "w") as f:
        f.write(text)
    log = compare(E.Problem(E.parse_input(workdir + "/input.txt"), workdir))
    assert max(np.abs(o["tabs"]).max() for o in log) > 0 and max(np.abs(o["EF_probe"]).max() for o in log) > 0


# Hermitian dipoles, whose lower elements are the conjugates
@pytest.mark.parametrize("nb,n", [((1, 1), 12), ((1, 2), 40)])
def test_crystal_model_in_one_launch(workdir, nb, n):
    compare(E.Problem(E.parse_input(W.crystal(workdir, nb=nb, nkf=13, n=n, duration=2.0, t_fin_fs=0.6)), workdir))


def test_run_of_several_launches_keeps_the_history(workdir):
    """More steps than one launch takes: Adams-Bashforth's derivatives cross the gap."""
    pb = make(workdir, "hbn", 8, 8, "Adams_Bashforth 5\n", 500, t_fin=170.0)
    assert pb.info.nsteps > 1 << 14
    a, b = E.Context(pb), E.Context(pb, use_graphs=False)
    a.run()
    assert a.last_timing()[1] == 2
    b.run()
    assert np.abs(a.get_state() - b.get_state()).max() <= 1e-13
    assert len(a.obs()) == len(b.obs())


def test_runs_that_share_the_device(workdir):
    """Contexts in threads of their own beside a batch that advances: every run ends
    with the state of a run by itself."""
    pb = make(workdir, "hbn", 60, 60, "", 3)
    alone = E.Context(pb)
    alone.run()
    want, failed = alone.get_state(), []

    def runs(c):
        try:
            for _ in range(4):
                c.reset()
                c.run()
                assert np.abs(c.get_state() - want).max() <= 1e-13
        except Exception as e:  # noqa: BLE001 (reported below)
            failed.append(e)

    batch = E.Batch()
    slot = batch.add(make(workdir + "/b", "hbn", 48, 48, "", 5, t_fin=1.0))
    threads = [threading.Thread(target=runs, args=(c,)) for c in [E.Context(pb) for _ in range(3)]]
    for t in threads:
        t.start()
    while batch.poll(slot)[0] == abi.EDUS_INST_RUNNING:
        batch.advance(16)
    for t in threads:
        t.join()
    assert not failed, failed
