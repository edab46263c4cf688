"""Host paths over a stand-in CUDA runtime: calls that fail, work that shares a
device, devices other than the current one. No GPU needed."""
from host_paths import run_host


def test_state_is_read_from_a_device_that_is_not_the_current_one(workdir):
    """The layout kernel and its buffer belong to the context's device."""
    run_host(workdir, """
    pb = problem(W.hbn_rk4(d + "/a", n=8, t_fin_fs=0.1))
    a, b = E.Context(pb, device=1), E.Context(pb, device=0)  # device 0 is current now
    assert a.get_state().shape == (64, 3, 3) and b.get_state().shape == (64, 3, 3)
    """)
