"""The work that users of this package have it do, as cases that can be timed.

Every case is a whole use of a public entry point on synthetic input files:

  single  one solve in a context of its own (edus_b200.Context): reset, run,
          the observable log and the final density matrix
  batch   many solves in one edus_b200.Batch: admission, the run to the end of
          every time grid, the logs and final density matrices, release
  serve   requests sent to a running edus_b200.Server, until all are answered

Models are the ones of edus_b200.workloads: hBN (Haldane_CoreBN_Nedge, three
bands, two in batches once the decoupled core is dropped) and the seeded
synthetic Wannier model with 8 or 16 bands. Pulses are short (some fs at
1.6 eV) and end with the run, so every step sees a field. Grids are even, as
the k stencil needs them to be.

`exact` restates the equations of motion in complex128 torch, from the model's
formulas and the written model and table files.
"""
import math
import os
import random
import tempfile

import numpy as np
import torch

import edus_b200 as E
from edus_b200 import abi
from edus_b200 import workloads as W

FS = 1.0 / 0.02418884326505      # a.u. of time per fs
EV = 1.0 / 27.211396             # a.u. of energy per eV
BOHR = 1.0 / 0.52917721092       # bohr per Angstrom
PHOTON_EV = 1.6
T_START = -0.21 * FS             # the reference's first instant
COULOMB_CAP = 20                 # Fourier modes of the packaged mean-field tables


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # the smallest solve: a convergence test's first grid; every step is launches and latency
        dict(name="hbn_24_rk4", form="single", kind="hbn", n1=24, n2=24, fs=1.0, dt=0.01, res=10, solver="rk4"),
        # the plain hBN run: 60 x 60, RK4, an output record at every step
        dict(name="hbn_60_rk4", form="single", kind="hbn", n1=60, n2=60, fs=3.0, dt=0.01, res=1, solver="rk4"),
        # the reference's example run: 70 x 70, Adams-Bashforth 5, circular pump, Gaussian probe on a decaying core hole
        dict(name="corehole_70_ab5", form="single", kind="corehole", n1=70, n2=70, fs=2.4, dt=0.002418884326505, res=5, solver="ab5"),
        # excitonic hBN: 120 x 120 with the Rytova-Keldysh mean field, Adams-Bashforth 4
        dict(name="coulomb_120_ab4", form="single", kind="coulomb", n1=120, n2=120, fs=3.0, dt=0.005, res=10, solver="ab4"),
        # an 8-band Wannier model on its production grid in FP64
        dict(name="wannier8_96_fp64", form="single", kind="wannier", nw=8, n1=96, n2=96, fs=2.0, dt=0.01, res=10, solver="rk4"),
        # a 16-band model on a coarse grid that is not a square
        dict(name="wannier16_30x34_fp64", form="single", kind="wannier", nw=16, n1=30, n2=34, fs=1.5, dt=0.01, res=10, solver="rk4"),
        # velocity gauge: H and D rebuilt for every stage on the tensor cores
        dict(name="vgauge8_64_mixed", form="single", kind="vgauge", nw=8, n1=64, n2=64, fs=1.0, dt=0.01, res=10, solver="rk4"),
        # one model under 16 pulses at once: a carrier-envelope scan in mixed precision
        dict(name="batch_wannier8_96_mixed", form="batch", kind="wannier", nw=8, count=16, nmin=96, nmax=96, fs=1.5, fs_max=1.5,
             dt=0.01, res=10, precision="mixed"),
        # the same with 16 bands, on smaller uneven grids
        dict(name="batch_wannier16_mixed", form="batch", kind="wannier", nw=16, count=6, nmin=48, nmax=72, fs=1.0, fs_max=1.4,
             dt=0.01, res=10, precision="mixed"),
        # a parameter sweep: half hBN, half 8-band Wannier, uneven grids and durations
        dict(name="sweep_mixed", form="batch", kind="sweep", nw=8, count=24, nmin=48, nmax=144, fs=1.0, fs_max=2.0,
             dt=0.01, res=10, precision="mixed"),
        # the same sweep, smaller, in FP64 (the default precision of a batch)
        dict(name="sweep_fp64", form="batch", kind="sweep", nw=8, count=10, nmin=48, nmax=112, fs=1.0, fs_max=2.0,
             dt=0.01, res=10, precision="fp64"),
        # a served stream: hBN, 8-band and mean-field requests that arrive together
        dict(name="serve_mixed", form="serve", kind="stream", nw=8, count=9, nmin=36, nmax=96, fs=1.0, fs_max=2.0,
             dt=0.01, res=10, precision="mixed"),
    ]


def _even(rng, lo, hi):
    return 2 * round(math.exp(rng.uniform(math.log(lo / 2), math.log(hi / 2))))


def draw(rng):
    """One more case: any listed use, with sizes over its range."""
    kind = rng.choice(["hbn", "hbn", "corehole", "coulomb", "wannier", "vgauge", "batch", "batch16", "sweep", "sweep64", "stream"])
    if kind in ("hbn", "corehole", "coulomb"):
        n1 = _even(rng, 16, 120)
        n2 = n1 if rng.random() < 0.5 else min(128, n1 + 2 * rng.randint(0, 8))
        c = dict(form="single", kind=kind, n1=n1, n2=n2, fs=round(rng.uniform(0.6, 2.0), 2), dt=0.01, res=rng.choice([1, 5, 10]))
        c["solver"] = {"hbn": "rk4", "corehole": "ab5", "coulomb": rng.choice(["ab4", "ab4", "rk4"])}[kind]
        if kind == "corehole":
            c["dt"] = 0.002418884326505
        elif kind == "coulomb":
            c["dt"] = 0.005
        return c
    if kind == "wannier":
        nw = rng.choice([2, 8, 8, 16])
        n1 = _even(rng, 12, 36 if nw == 16 else 80)
        n2 = n1 if rng.random() < 0.5 else n1 + 2 * rng.randint(0, 4)
        return dict(form="single", kind="wannier", nw=nw, n1=n1, n2=n2, fs=round(rng.uniform(0.6, 1.5), 2), dt=0.01, res=10, solver="rk4")
    if kind == "vgauge":
        n = _even(rng, 24, 64)
        return dict(form="single", kind="vgauge", nw=8, n1=n, n2=n, fs=round(rng.uniform(0.5, 1.0), 2), dt=0.01, res=10, solver="rk4")
    if kind in ("batch", "batch16"):
        nw = 16 if kind == "batch16" else 8
        hi = _even(rng, 40, 60 if nw == 16 else 96)
        return dict(form="batch", kind="wannier", nw=nw, count=rng.randint(2, 5 if nw == 16 else 14), nmin=max(32, hi - 2 * rng.randint(0, 12)),
                    nmax=hi, fs=0.8, fs_max=round(rng.uniform(0.8, 1.4), 2), dt=0.01, res=10, precision=rng.choice(["mixed", "mixed", "fp64"]) if nw == 8 else "mixed")
    hi = _even(rng, 64, 112)
    common = dict(nw=8, nmin=40, nmax=hi, fs=0.8, fs_max=round(rng.uniform(1.0, 1.8), 2), dt=0.01, res=10)
    if kind == "stream":
        return dict(form="serve", kind="stream", count=rng.randint(4, 9), precision="mixed", **dict(common, nmin=36, nmax=min(hi, 96)))
    return dict(form="batch", kind="sweep", count=rng.randint(4, 16 if kind == "sweep" else 10),
                precision="mixed" if kind == "sweep" else "fp64", **common)


# ------------------------------------------------------------------ inputs

def _between(fs, dt):
    """A duration near fs that ends between two steps, so that no rounding decides on the last one."""
    return round((round((fs + 0.21) / dt) + 0.4) * dt - 0.21, 9)


def _specs(case, seed):
    """The solves of a case: one dict each, from the seed alone."""
    rng = random.Random(f"edus {seed}")

    def pulse():
        return dict(field=rng.uniform(0.2, 0.6), phase=rng.uniform(0.0, 2 * math.pi), gap=rng.uniform(5.4, 6.2), t1=rng.uniform(2.2, 2.4))

    model = rng.randrange(1, 1 << 30)
    if case["form"] == "single":
        s = dict(kind=case["kind"], n1=case["n1"], n2=case["n2"], fs=_between(case["fs"], case["dt"]), solver=case["solver"], seed=model, **pulse())
        return [dict(s, nw=case.get("nw", 3), dt=case["dt"], res=case["res"])]
    out = []
    for i in range(case["count"]):
        kind = case["kind"]
        if kind == "sweep":
            kind = "hbn" if i % 2 == 0 else "wannier"
        elif kind == "stream":
            kind = ("hbn", "wannier", "coulomb")[i % 3]
        # sizes and durations are spread evenly over their ranges, so that every seed has the same work
        f = i / max(1, case["count"] - 1)
        n = 2 * round((case["nmin"] + f * (case["nmax"] - case["nmin"])) / 2)
        fs = case["fs"] + ((i * 7) % case["count"]) / case["count"] * (case["fs_max"] - case["fs"])
        dt = 0.005 if kind == "coulomb" else case["dt"]
        out.append(dict(kind=kind, n1=n, n2=n, fs=_between(fs, dt), solver="ab4" if kind == "coulomb" else "rk4", seed=model,
                        nw=case["nw"] if kind == "wannier" else 3 if kind == "coulomb" else 2, dt=dt, res=case["res"], **pulse()))
    return out


def _model_file(root, s):
    path = os.path.join(root, f"W{s['nw']}_tb.dat")
    if not os.path.exists(path):
        W.write_wannier_tb(path, nw=s["nw"], seed=s["seed"])
    return path


def _write(root, s, i):
    """input.txt and its model or table files in a directory of their own."""
    d = os.path.join(root, f"i{i}")
    os.makedirs(d, exist_ok=True)
    common = dict(n=s["n1"], field=s["field"], photon=PHOTON_EV, duration=s["fs"], dt_fs=s["dt"], it_res=s["res"], phase=s["phase"])
    if s["kind"] == "hbn":
        path = W.hbn_rk4(d, gap=s["gap"], t1=s["t1"], **common)
    elif s["kind"] == "coulomb":
        path = W.hbn_coulomb(d, rk4=s["solver"] == "rk4", **common)
    elif s["kind"] == "corehole":
        e0 = s["field"] * 1e10 / 5.14221e11
        path = os.path.join(d, "input.txt")
        with open(path, "w") as f:
            f.write("CORE\n\ntdse{\n"
                    f"tightbinding Haldane_CoreBN_Nedge gap= {s['gap']} t1= {-s['t1']} t2= 0 phi0= 0\n"
                    f"dt {s['dt'] * FS:.12g} au\nt_fin {s['fs'] * FS:.12g} au\nAdams_Bashforth 5\n}}\n\n"
                    "nkpt{\n1 0 0\n}\n\ndecoherence{\ncorehole 0.00396892 au\n}\n\n"
                    f"laserpump sin2 {{\nfrequency {PHOTON_EV * EV:.12g}\nintensity {e0 * e0 * 3.51e16:.12g} wcm2\n"
                    f"cycles {s['fs'] * FS * PHOTON_EV * EV / (2 * math.pi):.12g}\npolarization circular 0 1 0 0 0 1\n"
                    f"phase {s['phase']:.12g}\n}}\n\n"
                    "laserprobe gaussian {\nsigma 0.08 fs\ndelay 0 fs\nintensity 10.e+06\nfrequency 15.06\npolarization 1 0 0\n}\n\n"
                    f"observables{{\nit_resolution {s['res']}\nTAbs\nCurrent\n}}\n")
    else:
        os.symlink(_model_file(root, s), os.path.join(d, f"W{s['nw']}_tb.dat"))
        path = W.wannier(d, nw=s["nw"], name=f"W{s['nw']}", write_model=False, **common)
    with open(path) as f:
        text = f.read()
    head, tail = text.split("nkpt{\n", 1)
    text = head + f"nkpt{{\n1 {s['n1']} {s['n2']}\n" + tail.split("\n", 1)[1]
    if s["kind"] == "vgauge":
        text = text.replace("tdse{\nWannier\n", "tdse{\nWannier\nvelocity_gauge\n")
    with open(path, "w") as f:
        f.write(text)
    return path, d


class _State:
    """What a user's program keeps between calls; its directory goes with it."""

    def __init__(self):
        self.dir = tempfile.TemporaryDirectory(prefix="edus_case_")
        self.open = []

    def __del__(self):
        for x in reversed(self.open):
            x.close()
        self.dir.cleanup()


def prepare(case, seed):
    st = _State()
    st.form = case["form"]
    specs = _specs(case, seed)
    files = [_write(st.dir.name, s, i) for i, s in enumerate(specs)]
    prec = abi.EDUS_PREC_MIXED if case.get("precision") == "mixed" or case["kind"] == "vgauge" else abi.EDUS_PREC_FP64
    if st.form == "single":
        path, d = files[0]
        pb = E.Problem(E.parse_input(path), d)
        st.ctx = E.Context(pb, precision=prec)
        st.open = [pb, st.ctx]
    elif st.form == "batch":
        st.problems = []
        for s, (path, d) in zip(specs, files):
            pb = E.Problem(E.parse_input(path), d, defer_model=s["kind"] == "wannier")
            st.problems.append(pb.drop_decoupled_core() if s["kind"] == "hbn" else pb)
        st.batch = E.Batch(precision=prec, max_instances=max(64, len(specs)))
        st.open = st.problems + [st.batch]
    else:
        st.requests = [(E.parse_input(path), d) for path, d in files]
        st.server = E.Server(precision=prec)
        st.open = [st.server]
    return st


# ------------------------------------------------------------------ one pass

def _log(obs):
    return {q: np.array([o[q] for o in obs]) for q in ("t", "J1", "J2", "pol", "pop", "tabs")}


def run(state):
    if state.form == "single":
        c = state.ctx
        c.reset()
        c.run()
        return dict(_log(c.obs()), state=c.get_state())
    if state.form == "batch":
        b = state.batch
        slots = [b.add(pb) for pb in state.problems]
        while any(b.poll(q)[0] != abi.EDUS_INST_DONE for q in slots):
            b.advance(64)
        logs = [_log(b.obs(q)) for q in slots]
        rho = [b.get_state(q) for q in slots]
        for q in slots:
            b.release(q)
        return dict(_joined(logs), state=rho)
    s = state.server
    ids = [s.submit(p, d) for p, d in state.requests]
    s.drain(120.0)
    logs = [_log(s.obs(r)) for r in ids]
    for r in ids:
        s.forget(r)
    return _joined(logs)


def _joined(logs):
    """The logs of several solves, one after the other, by quantity and band count."""
    out = {}
    for g in logs:
        n = g["pop"].shape[1]
        for q, v in g.items():
            out.setdefault(f"{q}{n}", []).append(v)
    return {q: np.concatenate(v) for q, v in out.items()}


def _steps(s):
    return int((s["fs"] * FS - T_START) / (s["dt"] * FS)) + 1


def work(case):
    """The tables and the state read once, the log and the state written once;
    commutator, k-gradient and update of every right-hand side."""
    flops = size = 0.0
    for s in _specs(case, 0):
        n, nk, steps = s["nw"], s["n1"] * s["n2"], _steps(s)
        if case["kind"] in ("hbn", "corehole"):
            n = 3
        tri = n * (n + 1) / 2
        rhs = 4 if s["solver"] == "rk4" else 1
        per = 8.0 * n ** 3 + tri * (4 * 6 + 16)
        if s["kind"] == "coulomb":
            per += tri * 4 * (2 * COULOMB_CAP) * 2  # truncated transform there and back, separable
        if s["kind"] == "vgauge":
            per += 4 * tri * 121 * 8  # Fourier sums of H and D at k + A
        flops += rhs * steps * nk * per
        # state, H and three components of D as upper triangles, U; the state and the records out
        size += nk * 16.0 * (tri * 5 + 2 * n * n) + (steps / s["res"]) * 400
    return {"bytes": size, "flops": flops}


# ------------------------------------------------------------------ the same in 64 bits

_C = torch.complex128


def _text(x):
    """a number as the input files carry it"""
    return float(f"{x:.12g}")


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Exact:
    """The equations of motion of one solve on a k grid [n1, n2]."""

    def __init__(self, s, d, core):
        self.s, self.dev = s, _device()
        n1, n2 = s["n1"], s["n2"]
        self.core = core
        self.wannier = s["kind"] in ("wannier", "vgauge")
        if self.wannier:
            a = np.diag([10.0, 2.5, 2.5]) * BOHR
        else:
            lc, ang = 2.5 * BOHR, math.pi / 6
            a = np.array([[6.33031, 0, 0], [0, lc * math.cos(ang), lc * math.sin(ang)], [0, lc * math.cos(ang), -lc * math.sin(ang)]])
        self.a = a
        self.b = 2 * math.pi * np.linalg.inv(a).T
        self.k1 = -0.5 + np.arange(n1) / n1
        self.k2 = -0.5 + np.arange(n2) / n2
        self._stencil()
        g1, g2 = np.meshgrid(self.k1, self.k2, indexing="ij")
        if self.wannier:
            self._read_wannier(os.path.join(d, f"W{s['nw']}_tb.dat"))
            self.H, self.D = self.tables(0.0, 0.0)
            self.U = self._vectors(self.H)
            self.n, self.filled = s["nw"], s["nw"] // 2
        else:
            self._hbn(g1, g2)
        n = self.n
        self.P0 = torch.einsum("xyia,xyib->xyab", self.U[:, :, : self.filled], self.U[:, :, : self.filled].conj())
        self.off = self._core_mask()
        if s["kind"] == "coulomb":
            self._mean_field(d)

    def _t(self, x):
        return torch.as_tensor(np.asarray(x), dtype=_C, device=self.dev)

    # shells of equal |b| around k = 0 until the weights reproduce the gradient
    def _stencil(self):
        n1, n2 = self.s["n1"], self.s["n2"]
        pts = [(i, j) for i in range(n1) for j in range(n2)]
        kc = np.array([[0.0, self.k1[i], self.k2[j]] for i, j in pts]) @ self.b
        r = np.linalg.norm(kc, axis=1)
        seen, shells = 1e-8, []
        sel = [(x, y, z, w) for x in range(3) for y in range(x, 3) for z in range(y, 3) for w in range(z, 3)]
        while True:
            rad = r[r > seen + 1e-11].min()
            seen = rad
            shells.append(np.nonzero(np.abs(r - rad) < 1e-11)[0])
            A = np.zeros((21, len(shells)))
            for c, idx in enumerate(shells):
                b = kc[idx]
                A[0, c], A[1, c], A[2, c] = (b[:, 1] ** 2).sum(), (b[:, 2] ** 2).sum(), (b[:, 1] * b[:, 2]).sum()
                for q, (x, y, z, w) in enumerate(sel):
                    A[5 + q, c] += (b[:, x] * b[:, y] * b[:, z] * b[:, w]).sum()
            q = np.zeros(21)
            q[:2] = 1
            w = np.linalg.pinv(A, rcond=1e-16) @ q
            if np.linalg.norm(A @ w - q) < 1e-7:
                break
        self.steps = []
        for c, idx in enumerate(shells):
            for i in idx:
                d1, d2 = round(kc[i] @ self.a[1] / (2 * math.pi) * n1), round(kc[i] @ self.a[2] / (2 * math.pi) * n2)
                self.steps.append((d1, d2, w[c] * kc[i]))

    def gradient(self, f, E):
        """sum_b w_b (E . b) f(k + b)"""
        out = torch.zeros_like(f)
        for d1, d2, wb in self.steps:
            out += float(wb @ E) * torch.roll(f, (-d1, -d2), (0, 1))
        return out

    def _hbn(self, g1, g2):
        s = self.s
        gap, t1 = s["gap"] * EV, (-s["t1"] if s["kind"] == "corehole" else s["t1"]) * EV
        if s["kind"] == "coulomb":
            gap, t1 = 5.8 * EV, 2.3 * EV
        f = 1.0 + np.exp(-2j * math.pi * g1) + np.exp(-2j * math.pi * g2)
        H = np.zeros(g1.shape + (3, 3), complex)
        H[..., 0, 0], H[..., 1, 1], H[..., 2, 2] = -15.06, -gap / 2, gap / 2
        H[..., 1, 2], H[..., 2, 1] = t1 * f, t1 * f.conj()
        B = t1 * f
        mod = np.sqrt(np.abs(B) ** 2 + gap * gap / 4)
        half = np.angle(B.conj()) / 2
        up, dn = np.sqrt((mod - gap / 2) / 2 / mod), np.sqrt((mod + gap / 2) / 2 / mod)
        U = np.zeros_like(H)
        U[..., 0, 0] = 1
        U[..., 1, 1], U[..., 1, 2] = np.exp(1j * half) * dn, -np.exp(-1j * half) * up
        U[..., 2, 1], U[..., 2, 2] = np.exp(1j * half) * up, np.exp(-1j * half) * dn
        D = np.zeros((3, 3, 3))
        D[0, 0, 1] = D[0, 1, 0] = 0.0697595094
        D[1, 2, 2] = 2.5 * BOHR / math.sqrt(3.0)
        lo = 0 if self.core else 1
        self.H, self.U = self._t(H[..., lo:, lo:]), self._t(U[..., lo:, lo:])
        self.D = self._t(D[:, lo:, lo:])[:, None, None].expand(3, s["n1"], s["n2"], 3 - lo, 3 - lo)
        self.n, self.filled = 3 - lo, 2 - lo

    def _read_wannier(self, path):
        with open(path) as f:
            tok = "".join(f.readlines()[4:]).split()
        nw, nr = int(tok[0]), int(tok[1])
        v = np.array(tok[2 + nr:], float)
        deg = np.array(tok[2: 2 + nr], float)[:, None, None]
        h = v[: nr * (3 + 4 * nw * nw)].reshape(nr, -1)
        r = v[nr * (3 + 4 * nw * nw):].reshape(nr, -1)
        h4, r8 = h[:, 3:].reshape(nr, nw, nw, 4), r[:, 3:].reshape(nr, nw, nw, 8)
        # the file runs over the second index first
        HR = (h4[..., 2] + 1j * h4[..., 3]).transpose(0, 2, 1) / deg * EV
        XR = [(r8[..., 2 + 2 * x] + 1j * r8[..., 3 + 2 * x]).transpose(0, 2, 1) / deg * BOHR for x in range(3)]
        self.R = torch.as_tensor(h[:, 1:3].copy(), dtype=torch.float64, device=self.dev)
        self.coef = self._t(np.stack([HR] + XR, 1)).reshape(nr, -1)
        self.nw = nw

    def tables(self, A1, A2):
        """H, D of the Wannier model at k + A (crystal coordinates)."""
        n1, n2, nw = self.s["n1"], self.s["n2"], self.nw
        k1 = torch.as_tensor(self.k1 + A1, device=self.dev)
        k2 = torch.as_tensor(self.k2 + A2, device=self.dev)
        p1 = torch.exp(2j * math.pi * torch.outer(k1, self.R[:, 0]).to(_C))
        p2 = torch.exp(2j * math.pi * torch.outer(k2, self.R[:, 1]).to(_C))
        X = ((p1[:, None, :] * p2[None, :, :]).reshape(n1 * n2, -1) @ self.coef).reshape(n1, n2, 4, nw, nw)
        H = X[:, :, 0].clone()
        H.diagonal(dim1=-2, dim2=-1).imag.zero_()
        H = torch.triu(H) + torch.triu(H, 1).mH
        D = X[:, :, 1:].clone()
        D.diagonal(dim1=-2, dim2=-1).imag.zero_()
        return H, (0.5 * (D + D.mT)).permute(2, 0, 1, 3, 4).contiguous()

    def _vectors(self, H):
        """rows: the conjugated eigenvectors, ascending energies"""
        return torch.linalg.eigh(H)[1].mH

    # ---- field
    def field(self, t):
        s = self.s
        e0 = s["field"] * 1e10 / 5.14221e11
        wl = _text(PHOTON_EV * EV)
        e0 = math.sqrt(_text(e0 * e0 * 3.51e16) / 3.51e16)
        tf = _text(s["fs"] * FS * PHOTON_EV * EV / (2 * math.pi)) * (2 * math.pi / wl)
        env = e0 * math.sin(math.pi * t / tf) ** 2 if 0 <= t <= tf else 0.0
        a, b = (fn(wl * t + _text(s["phase"])) for fn in (math.sin, math.cos))
        if s["kind"] != "corehole":
            return np.array([0, 0, env * a]), np.zeros(3)
        sig = 0.08 * FS
        # centred as the reference does it after a sin2 pump: on half the pump, less sigma / 2 probe periods
        d = t - (tf / 2 - sig / 2 * (2 * math.pi / 15.06))
        pe = math.sqrt(10.0e6 / 3.51e16) * math.exp(-d * d / (2 * sig * sig)) if d * d < 40 * sig * sig else 0.0
        return np.array([0, env * a, env * b]), np.array([0.5 * pe, 0, 0])  # the probe in its rotating frame

    def _core_mask(self):
        m = torch.zeros(self.n, self.n, dtype=_C, device=self.dev)
        if not self.wannier and self.core:
            m[0, 1:] = 1
            m[1:, 0] = 1
        return m

    # ---- mean field: truncated Fourier series of rho against the tables on file
    def _mean_field(self, d):
        c = os.path.join(d, "Output", "Coulomb")

        def rows(name):
            v = np.loadtxt(os.path.join(c, f"{name}{W.COULOMB_LABEL}.txt"))
            return v[:, 0::2] + 1j * v[:, 1::2]

        nc, n = COULOMB_CAP, self.n
        up = np.triu(np.ones((n, n)))
        co = []
        for q in "ABCD":
            v = rows(f"{q}_coeff").reshape(nc, nc, n, n)
            v[..., range(n), range(n)] = v[..., :1, 0] if q in "AD" else 0.0
            co.append(self._t(v * up))
        self.co = co
        s = rows("Screen_const_").reshape(n, n)
        s[range(n), range(n)] = s[0, 0]
        self.screen = self._t(np.triu(s.conj()))
        self.VH = self._t(np.loadtxt(os.path.join(c, f"V_Hartree_{W.COULOMB_LABEL}.txt")))
        m = np.arange(nc)
        self.tr = [self._t(fn(2 * math.pi * np.outer(m, k))) for k in (self.k1, self.k2) for fn in (np.cos, np.sin)]
        nk = self.s["n1"] * self.s["n2"]
        self.corr = self._t((1 - 4 * math.pi ** 2 * (m[:, None] ** 2 + m[None, :] ** 2) / (27.0 * nk)) / nk)[..., None, None]
        self.X0 = self._modes(self.P0)
        self.ncond = 0.0

    def _modes(self, P):
        c1, s1, c2, s2 = self.tr
        A, B, C, D = self.co

        def tf(u, v):
            return self.corr * torch.einsum("mx,ny,xyij->mnij", u, v, P)

        cc, cs, sc, ss = tf(c1, c2), tf(c1, s2), tf(s1, c2), tf(s1, s2)
        eh = (self.VH @ cc[0, 0].diagonal().real.to(_C)).real
        return (A * cc + D * ss + B * cs + C * sc, A * cs - D * sc - B * cc + C * ss,
                A * sc - D * cs + B * ss - C * cc, A * ss + D * cc - B * sc - C * cs, eh)

    def hamiltonian(self, P):
        if self.s["kind"] != "coulomb":
            return self.H
        c1, s1, c2, s2 = self.tr
        f = [x - x0 for x, x0 in zip(self._modes(P), self.X0)]
        X = sum(torch.einsum("mx,ny,mnij->xyij", u, v, y) for u, v, y in ((c1, c2, f[0]), (c1, s2, f[1]), (s1, c2, f[2]), (s1, s2, f[3])))
        X = -X.conj()
        if self.ncond > 1e-20:
            X = X - self.screen * (P - self.P0).conj()
        X = torch.triu(X, 1) + torch.diag_embed(X.diagonal(dim1=-2, dim2=-1).real.to(_C) + f[4].to(_C))
        return self.H + X + torch.triu(X, 1).mH

    # ---- equations of motion
    def rhs(self, P, EF, grad):
        s = self.s
        self.Hr = H = self.hamiltonian(P)
        pump = sum(float(EF[0][x]) * self.D[x] for x in range(3) if EF[0][x])
        if isinstance(pump, torch.Tensor):
            H = H + pump * (1 - self.off)
        if EF[1].any():
            H = H + sum(float(EF[1][x]) * self.D[x] for x in range(3) if EF[1][x]) * self.off
        C = P @ H.mT
        v = -1j * (C - C.mH)
        if s["kind"] == "corehole":
            w = torch.zeros(3, 3, dtype=_C, device=self.dev)
            w[0, 1:] = 15.06j
            v = v + w * P + (w * P).mH
            v = v + self._decay(P)
        if grad:
            v = v + self.gradient(P, EF[0])
        return v

    def _decay(self, P):
        T = torch.zeros(3, 3, dtype=_C, device=self.dev)
        T[0, :] = T[:, 0] = 0.00396892 / 2
        T[0, 0] = 0.00396892
        U = self.U
        M = T * (U.conj() @ P @ U.mT)
        v = -torch.einsum("xyjb,xyia,xyab->xyij", U.mH, U.conj(), M)
        v = v + torch.einsum("xyqj,xyqi,q->xyij", U[:, :, :2].conj(), U[:, :, :2], T.diagonal()[:2])
        v = torch.triu(v, 1) + torch.diag_embed(v.diagonal(dim1=-2, dim2=-1).real.to(_C))
        return v + torch.triu(v, 1).mH

    def at_A(self, t0, t):
        """vector potential gained from t0 to t (Gauss-Legendre, eight points)"""
        x, w = np.polynomial.legendre.leggauss(8)
        h, m = 0.5 * (t - t0), 0.5 * (t + t0)
        return -h * sum(wi * self.field(m + h * xi)[0] for xi, wi in zip(x, w))

    def observe(self, P):
        s, n = self.s, self.n
        nk = s["n1"] * s["n2"]
        H = self.Hr if s["kind"] == "coulomb" else self.H
        U = self._vectors(H) if s["kind"] in ("coulomb", "vgauge") else self.U
        pop = torch.einsum("xyci,xyij,xycj->xyc", U.conj(), P, U).real.mean((0, 1))
        pop[: self.filled] = 1 - pop[: self.filled]
        if s["kind"] == "coulomb":  # (before the pulse this is rounding noise on every side)
            self.ncond = float(pop.max().clamp(min=0))
        cross = abs(np.linalg.det(self.a[1:, 1:]))
        scale = 1.0 / nk / cross
        ge = torch.zeros((3,) + H.shape, dtype=_C, device=self.dev)
        for d1, d2, wb in self.steps:
            dH = torch.roll(H, (-d1, -d2), (0, 1)) - H
            for x in (1, 2):
                ge[x] += float(wb[x]) * dH
        J1 = (ge * P).sum((1, 2, 3, 4)) * scale
        J2 = -2 * torch.einsum("xyil,dxyil->d", H, P @ self.D.conj()).imag * scale
        pol = torch.einsum("dxyij,xyij->d", self.D, P) / nk
        tabs = torch.zeros(3, dtype=_C, device=self.dev)
        if s["kind"] == "corehole":
            vol = abs(np.linalg.det(self.b)) / nk
            tabs = -2 * (self.D[:, :, :, 0, 1:] * P[None, :, :, 0, 1:]).sum((1, 2, 3)) * (vol / nk)
        return {"J1": J1, "J2": J2, "pol": pol, "pop": pop, "tabs": tabs}

    def solve(self):
        s = self.s
        dt, t, P = s["dt"] * FS, T_START, self.P0.clone()
        self.Hr = self.H
        order = int(s["solver"][2]) if s["solver"].startswith("ab") else 0
        coef = {4: [55 / 24, -59 / 24, 37 / 24, -9 / 24], 5: [1901 / 720, -2774 / 720, 2616 / 720, -1274 / 720, 251 / 720]}.get(order)
        ring, log, grad, A = [], [], True, np.zeros(3)
        vg = s["kind"] == "vgauge"

        def on(EF):
            return math.sqrt((EF[0] ** 2).sum() + (EF[1] ** 2).sum()) > 1e-20

        def move(ta, tb):
            nonlocal A
            if vg:
                A = A + self.at_A(ta, tb)
                c = self.a @ A / (2 * math.pi)
                self.H, self.D = self.tables(c[1], c[2])

        for it in range(_steps(s)):
            if it % s["res"] == 0:
                log.append(dict(t=t, **{q: v.cpu().numpy() for q, v in self.observe(P).items()}))
            E0 = self.field(t)
            if order and (s["kind"] != "coulomb" or it >= order - 1):
                k1 = self.rhs(P, E0, on(E0))
                ring = [k1] + ring[: order - 1]
                P = P + dt * sum(c * r for c, r in zip(coef, ring))
            else:
                Eh, E1 = self.field(t + dt / 2), self.field(t + dt)
                g = False if vg else on(E0) if order else grad
                k1 = self.rhs(P, E0, g)
                move(t, t + dt / 2)
                k2 = self.rhs(P + dt / 2 * k1, Eh, g)
                k3 = self.rhs(P + dt / 2 * k2, Eh, g)
                move(t + dt / 2, t + dt)
                k4 = self.rhs(P + dt * k3, E1, g)
                P = P + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
                grad = on(E1)
                if order:
                    ring = [k1] + ring[: order - 1]
            t += dt
        out = {q: np.array([o[q] for o in log]) for q in log[0]}
        return out, P.reshape(-1, self.n, self.n).cpu().numpy()


def exact(case, seed):
    with tempfile.TemporaryDirectory(prefix="edus_exact_") as root:
        logs, states = [], []
        for i, s in enumerate(_specs(case, seed)):
            if case["form"] == "single" and s["kind"] == "hbn":
                s["nw"] = 3
            _, d = _write(root, s, i)
            out, rho = _Exact(s, d, core=case["form"] == "single" or s["kind"] == "coulomb").solve()
            if case["form"] == "single":
                return dict(out, state=rho)
            logs.append(out)
            states.append(rho)
    return dict(_joined(logs), **({"state": states} if case["form"] == "batch" else {}))
