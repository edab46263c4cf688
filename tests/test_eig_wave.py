"""Velocity-gauge observables of 8 and 16 bands where the spectrum is a hard one for the
Jacobi eigensolver: every eigenvalue twice (the split is rounding noise), and a diagonal
H(k) at zero field (no rotation at all, eigenvalues out of order), against the oracle. The
population of a degenerate pair does not depend on its basis."""
import numpy as np
import pytest

import edus_b200 as E
from edus_b200 import workloads as W
from oracle_lib import Oracle

pytestmark = pytest.mark.gpu


def rewrite(path, nw, kind):
    """The model of `path` (nw / 2 orbitals) as Q (A + A) Q^T of nw orbitals, or the diagonal of its H."""
    lines = open(path).read().split("\n")
    half, nr = int(lines[4]), int(lines[5])
    rows = [l for l in lines[6 + (nr + 14) // 15:] if l.strip()]
    rng = np.random.Generator(np.random.PCG64(7))
    q = np.linalg.qr(rng.standard_normal((nw, nw)))[0]
    out = lines[:4] + [str(nw)] + lines[5:6 + (nr + 14) // 15]
    for i in range(2 * nr):
        block = rows[i * (1 + half * half): (i + 1) * (1 + half * half)]
        v = np.array([[float(x) for x in l.split()[2:]] for l in block[1:]])
        a = (v[:, 0::2] + 1j * v[:, 1::2]).T.reshape(-1, half, half).transpose(0, 2, 1)  # [comp][m][n]
        big = np.zeros((a.shape[0], nw, nw), complex)
        if kind == "pairs":
            big[:, :half, :half] = big[:, half:, half:] = a
            big = q @ big @ q.T
        elif i < nr and not any(int(x) for x in block[0].split()):
            big[0] = np.diag(rng.permutation(np.linspace(-1.5, 1.5, nw)))
        out += ["", block[0]]
        out += [f"{m + 1} {n + 1} " + " ".join(f"{c.real:.16e} {c.imag:.16e}" for c in big[:, m, n]) for n in range(nw) for m in range(nw)]
    with open(path, "w") as f:
        f.write("\n".join(out) + "\n")


@pytest.mark.parametrize("kind", ["pairs", "diagonal"])
@pytest.mark.parametrize("nw", [8, 16])
def test_populations_of_hard_spectra(workdir, nw, kind):
    W.write_wannier_tb(f"{workdir}/W_tb.dat", nw=nw // 2, nside=3)
    rewrite(f"{workdir}/W_tb.dat", nw, kind)
    path = W.wannier(workdir, nw=nw, nside=3, n=10, field=0.5, t_fin_fs=0.1, it_res=2, name="W", write_model=False)
    text = open(path).read().replace("Wannier\n", "Wannier\nvelocity_gauge\n")
    with open(path, "w") as f:
        f.write(text)
    p = E.parse_input(path)
    ctx = E.Context(E.Problem(p, workdir))
    ctx.run()
    got, want = ctx.obs(), Oracle(p, workdir).run()
    assert len(got) == len(want)
    for g, w in zip(got, want):
        a, b = np.array(g["pop"])[:nw], np.array(w["pop"])[:nw]
        if kind == "pairs":
            a, b = a[0::2] + a[1::2], b[0::2] + b[1::2]
        # means over k of values near 1, the bar of the other tests; two of them for a pair
        assert np.abs(a - b).max() <= 2e-13
    a, b = np.array([g["J1"] for g in got]), np.array([w["J1"] for w in want])
    assert np.abs(a - b).max() <= 1e-11 * max(np.abs(b).max(), 1e-4)
