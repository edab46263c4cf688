"""Host paths over a stand-in CUDA runtime: calls that fail, work that shares a
device, devices other than the current one. No GPU needed."""
import pytest

from host_paths import run_host


def test_state_is_read_from_a_device_that_is_not_the_current_one(workdir):
    """The layout kernel and its buffer belong to the context's device."""
    run_host(workdir, """
    pb = problem(W.hbn_rk4(d + "/a", n=8, t_fin_fs=0.1))
    a, b = E.Context(pb, device=1), E.Context(pb, device=0)  # device 0 is current now
    assert a.get_state().shape == (64, 3, 3) and b.get_state().shape == (64, 3, 3)
    """)


def test_whole_run_in_one_launch_only_where_nothing_else_is_at_work(workdir):
    """A context that begins while another call of the process works on the device
    takes the captured launch per stage; alone again, or on another device, one launch."""
    run_host(workdir, """
    hbn = problem(W.hbn_rk4(d + "/a", n=24, t_fin_fs=0.2))
    cou = problem(W.hbn_coulomb(d + "/c", n=12, t_fin_fs=0.1))
    a, b, far = E.Context(hbn), E.Context(hbn), E.Context(hbn, device=1)

    def run(c):
        F.fake_clear()
        g = F.fake_graph_launches()
        c.reset()
        c.run()
        assert c.clock()[0] == hbn.info.nsteps
        return launches("k_loop"), F.fake_graph_launches() - g

    @C.CFUNCTYPE(None)
    def others():  # in the first wait of a call
        F.fake_on_wait(None)
        seen.append((run(b), run(far)))

    def during(call):
        global seen
        seen = []
        F.fake_on_wait(others)
        call()
        assert len(seen) == 1
        return seen[0]

    shared = ((0, 1), (1, 0))
    assert run(b) == (1, 0)
    assert during(a.run) == shared          # a whole run
    a.reset()
    assert during(lambda: a.step(3)) == shared
    batch = E.Batch()
    batch.add(problem(W.hbn_rk4(d + "/b", n=12, t_fin_fs=0.2)))
    assert during(lambda: batch.advance(16)) == shared
    assert run(b) == (1, 0) and run(b) == (1, 0)
    slot = batch.add(cou)                    # runs by itself until it is polled
    assert run(b) == (0, 1)
    batch.advance(16)
    assert batch.poll(slot)[0] == abi.EDUS_INST_DONE
    assert run(b) == (1, 0)
    batch.add(cou)
    batch.close()                            # released without being polled
    assert run(b) == (1, 0)
    """)


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
def test_batch_without_layout_scratch(workdir, precision):
    """Device memory that is short: tables and states are laid out on the host (mixed
    precision keeps the state as a deviation from the ground state)."""
    run_host(workdir, """
    n, nk = 8, 100
    pb = problem(W.wannier(d + "/a", nw=n, nside=3, n=10, t_fin_fs=0.1, name="W"))
    limit("pool_refused", 48 * n * n * nk)      # scratch of the tables
    b = E.Batch(precision=abi.EDUS_PREC_%s)
    s = b.add(pb)
    limit("pool_refused", 16 * n * n * nk)      # the state's matrices
    got, P0 = b.get_state(s), pb.get("P0")
    assert launches("k_to_planes") == launches("k_from_planes") == 0
    assert np.array_equal(got, np.triu(P0) + np.conj(np.triu(P0, 1)).transpose(0, 2, 1))
    """ % precision)


def test_batch_state_without_pinned_buffers(workdir):
    """No pinned memory: a large state comes out through pageable memory."""
    run_host(workdir, """
    pb = problem(W.hbn_rk4(d + "/a", n=90, t_fin_fs=0.1))  # 1.2 MB of matrices
    b = E.Batch()
    s = b.add(pb)
    limit("pinned_max", 1024)
    assert b.get_state(s).shape == (8100, 3, 3)
    limit("pinned_max", 1 << 40)
    assert b.get_state(s).shape == (8100, 3, 3)
    """)


def test_states_of_one_batch_read_by_two_threads(workdir):
    """The pinned buffers serve one reader at a time. (Kernels do not run here: each
    reader's matrices are what its own device buffer holds, one byte all over.)"""
    run_host(workdir, """
    import threading
    pb = problem(W.hbn_rk4(d + "/a", n=90, t_fin_fs=0.1))  # 1.2 MB of matrices
    b = E.Batch()
    s, t = b.add(pb), b.add(pb)
    got = {}
    second = threading.Thread(target=lambda: got.update(second=b.get_state(t)))
    @C.CFUNCTYPE(None)
    def wait():  # the first reader's copy is on its way
        F.fake_on_wait(None)
        second.start()
        second.join(0.5)
    F.fake_on_wait(wait)
    got["first"] = b.get_state(s)
    second.join()
    one, two = (set(got[q].view(np.uint8).ravel()) for q in ("first", "second"))
    assert len(one) == len(two) == 1 and one != two
    """)


def test_tensor_core_sums_without_tensor_maps(workdir):
    """A driver that refuses the tensor maps: the sums run in the form that needs none."""
    run_host(workdir, """
    limit("encode_result", 1)
    path = W.wannier(d + "/v", nw=8, nside=3, n=8, t_fin_fs=0.1, name="W")
    text = open(path).read().replace("tdse{\\nWannier\\n", "tdse{\\nWannier\\nvelocity_gauge\\n")
    open(path, "w").write(text)
    c = E.Context(problem(path), precision=abi.EDUS_PREC_MIXED)
    assert launches("k_tc_gemmE") == 1 and launches("k_scatter64") == 1
    c.step(1)
    b = E.Batch(precision=abi.EDUS_PREC_MIXED)
    F.fake_clear()
    b.add(problem(W.wannier(d + "/b", nw=8, nside=3, n=8, t_fin_fs=0.1, name="W"), defer_model=True))
    assert launches("k_tc_gemmE") == 1 and launches("k_tc_planes") == 0 and launches("k_tc_gemm_tma") == 0
    limit("encode_result", 0)
    F.fake_clear()
    b.add(problem(W.wannier(d + "/b", nw=8, nside=3, n=8, t_fin_fs=0.1, name="W"), defer_model=True))
    assert launches("k_tc_planes") == 1 and launches("k_tc_gemmE") == 0
    """)


LAUNCH_COUNT = """
    def coulomb8(kind):
        # an 8-band Wannier model with small mean-field tables of two modes
        w, n, nc = d + "/" + kind, 8, 2
        path = W.wannier(w, nw=n, nside=3, n=8, t_fin_fs=0.2, it_res=2, name="W")
        os.makedirs(w + "/Output/Coulomb")
        for q in "ABCD":
            with open(f"{w}/Output/Coulomb/{q}_coefft.txt", "w") as f:
                f.write("1e-3 0 " * (nc * nc * n * n))
        with open(w + "/Output/Coulomb/Screen_const_t.txt", "w") as f:
            f.write("1e-3 0 " * (n * n))
        with open(w + "/Output/Coulomb/V_Hartree_t.txt", "w") as f:
            f.write("1e-3 " * (n * n))
        text = open(path).read()
        if kind == "adaptive":
            text = text.replace("tdse{\\n", "tdse{\\ndynamical_dt_evolution\\nepsStepAbs 0.001\\n")
        text += "\\nCoulomb{\\nqTF 0.01\\nNcut 2\\nepsilon_static 1.0\\nRytova_Keldysh\\nRead_Coulomb_from_files\\nlabelInput t\\n}\\n"
        open(path, "w").write(text)
        return path

    def vgauge():
        path = W.wannier(d + "/v", nw=8, nside=3, n=8, t_fin_fs=0.2, it_res=2, name="W")
        text = open(path).read().replace("tdse{\\nWannier\\n", "tdse{\\nWannier\\nvelocity_gauge\\n")
        open(path, "w").write(text)
        return path

    def adaptive3():
        return W.hbn_rk4(d + "/d", n=8, t_fin_fs=0.2, it_res=2, solver="dynamical_dt_evolution\\nepsStepAbs 0.001\\n")

    kind = "%s"
    path = dict(hbn=lambda: W.hbn_rk4(d + "/h", n=8, t_fin_fs=0.2, it_res=2), coulomb8=lambda: coulomb8("constant"),
                vgauge=vgauge, adaptive8=lambda: coulomb8("adaptive"), adaptive3=adaptive3)[kind]()
    prec = abi.EDUS_PREC_MIXED if kind == "vgauge" else abi.EDUS_PREC_FP64
    c = E.Context(problem(path), use_graphs=False, precision=prec)
    end = C.CFUNCTYPE(None)(F.fake_clear_flag)  # an adaptive run ends with the chunk that is waited for
    F.fake_on_wait(end)
    F.fake_clear()
    c.run()
    assert launches() > 0 and c.last_timing()[1] == launches()
"""


@pytest.mark.parametrize("kind", ["hbn", "coulomb8", "vgauge", "adaptive3", "adaptive8"])
def test_launch_count_is_the_number_of_launches(workdir, kind):
    run_host(workdir, LAUNCH_COUNT % kind)


@pytest.mark.parametrize("solver", ["", "Adams_Bashforth 4\\n"])
def test_whole_run_where_its_blocks_cannot_be_resident(workdir, solver):
    """A device that does not place a cluster of 16 blocks, or not all blocks at once: the
    cooperative grid instead of the cluster, and the launch per stage instead of both."""
    run_host(workdir, """
    def run(n):
        c = E.Context(problem(W.hbn_rk4(d + "/a", n=n, t_fin_fs=0.1, solver="%s")))
        F.fake_clear()
        c.run()
        assert c.clock()[0] > 0
        return launches("Li384ELb1E"), launches("Li384ELb0E"), launches("k_rhs_ep") > 0
    assert run(24) == (1, 0, False)     # one cluster
    assert run(60) == (0, 1, False)
    limit("max_clusters", 0)
    assert run(24) == (0, 1, False)
    limit("blocks_per_sm", 0)
    assert run(24) == (0, 0, True) and run(60) == (0, 0, True)
    limit("blocks_per_sm", 1)
    limit("max_clusters", 8)
    limit("sms", 1)                     # nothing left to step on beside the block that adds up
    assert run(24) == (0, 0, True)
    """ % solver)


def test_batch_accounts_for_the_memory_a_mean_field_state_is_read_through(workdir):
    run_host(workdir, """
    pb = problem(W.hbn_coulomb(d + "/a", n=24, t_fin_fs=0.1))
    b = E.Batch()
    before = F.fake_held()
    s = b.add(pb)
    b.advance(16)
    b.get_state(s)
    used = b.stats()["bytes_used"]
    assert used == F.fake_held() - before <= b.footprint(pb)
    b.release(s)
    used = b.stats()["bytes_used"]
    assert used == 0 and F.fake_held() == before
    """)
