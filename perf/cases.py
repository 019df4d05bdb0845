"""Performance cases: what users of this library have it do, at the sizes of
the repository's workloads (mdspherocyl_gb300/systems.py, bench.py), tests and
serving jobs, each through the public entry points.

listed() names the cases, draw() makes more of the same ranges, prepare() builds
the inputs and the handle a program keeps, run() makes one pass, work() counts
what a pass cannot do without, and exact() is the same pass in 64 bits with
plain torch, without this repository's code.
"""
from __future__ import annotations

import ctypes
import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from mdspherocyl_gb300 import lib as L
from mdspherocyl_gb300 import systems as S

DT = 1e-3
KEYS = "rpOlFT"
MU2 = 3.0
LATTICE_H = 0.5 * (200 * 1.001) / 32768  # spacing of the reference's real-space table

# what a case leaves out
DEFAULTS = {"nd": 1, "alpha": 6.0, "ksq": 36, "phi": 0.15, "rc": 0.0, "field": 0.0, "steps": 1, "systems": 1,
            "u_bond": 0.0, "species": 1, "bar_w": 0.1, "width": 480, "height": 480, "images": False}


def listed():
    return [
        # one small system between two outputs of its trajectory: the single-system
        # configuration of N = 256, the smallest run a user starts
        {"name": "steps_n256", "kind": "steps", "n": 256, "alpha": 5.6, "ksq": 27, "phi": 0.10, "steps": 50},
        # a program that keeps its state on the host and takes one step per call (the
        # bridge into the reference's driver), at an odd size: latency of one call
        {"name": "host_step_n333", "kind": "host_steps", "n": 333, "ksq": 27, "phi": 0.10, "steps": 1},
        # the reference's own boundary, one function after another, as its driver calls them
        {"name": "forces_n1000", "kind": "forces", "n": 1000, "alpha": 5.6, "ksq": 27, "phi": 0.12, "field": 1.0},
        # two off-centre dipoles per rod, a ragged size
        {"name": "steps_n1500_nd2", "kind": "steps", "n": 1500, "nd": 2, "steps": 20},
        # the N = 4096 configuration over all minimum-image pairs
        {"name": "steps_n4096", "kind": "steps", "n": 4096, "alpha": 7.0, "ksq": 64, "phi": 0.20, "steps": 20},
        # the same with its real-space cutoff
        {"name": "steps_n4096_rc", "kind": "steps", "n": 4096, "alpha": 7.0, "ksq": 64, "phi": 0.20, "rc": 3.5,
         "steps": 20},
        # the largest single system, in a field
        {"name": "steps_n32768", "kind": "steps", "n": 32768, "ksq": 100, "field": 2.0, "steps": 10},
        # its clustering by pair energy
        {"name": "clusters_n32768", "kind": "clusters", "n": 32768, "ksq": 100, "field": 2.0, "u_bond": 1.5},
        # many independent systems advanced together (the replica mix, N log-uniform in
        # [128, 2048]): the batched throughput
        {"name": "batch_64", "kind": "batch", "n": 2048, "n_lo": 128, "systems": 64, "steps": 10},
        # the pair-correlation histograms the driver accumulates, two species
        {"name": "correlations_n4096", "kind": "correlations", "n": 4096, "ksq": 27, "species": 2},
        # real-space forces on device buffers the caller owns (no allocation)
        {"name": "noalloc_n3001", "kind": "noalloc", "n": 3001},
        # a picture of the configuration
        {"name": "picture_n2000", "kind": "picture", "n": 2000, "ksq": 27, "phi": 0.10},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["steps", "steps", "steps", "host_steps", "forces", "batch", "clusters", "correlations",
                       "noalloc", "picture"])
    c = {"kind": kind, "alpha": round(rng.uniform(5.6, 7.0), 3), "ksq": rng.choice([27, 36, 64]),
         "phi": round(rng.uniform(0.05, 0.22), 3)}
    if kind == "steps":
        c["n"] = size(64, 16384)
        c["nd"] = 2 if c["n"] <= 4096 and rng.random() < 0.25 else 1
        if c["n"] >= 200 and rng.random() < 0.3:
            c["rc"] = 3.5
            c["phi"] = min(c["phi"], 0.20)
        if rng.random() < 0.3:
            c["field"] = round(rng.uniform(0.5, 2.0), 3)
        c["steps"] = max(4, min(50, 40000 // c["n"]))
    elif kind == "host_steps":
        c["n"] = size(64, 8192)
        c["steps"] = rng.choice([1, 1, 1, 2])
    elif kind == "forces":
        c["n"] = size(64, 8192)
        c["nd"] = 2 if c["n"] <= 2048 and rng.random() < 0.3 else 1
        c["field"] = rng.choice([0.0, 1.0])
    elif kind == "batch":
        c.update(n=2048, n_lo=rng.choice([64, 128]), systems=size(2, 64), steps=rng.randint(1, 10))
    elif kind == "clusters":
        c["n"] = size(256, 32768)
        c["u_bond"] = rng.choice([0.0, 1.5, round(rng.uniform(1.5, 2.5), 2)])
    elif kind == "correlations":
        c["n"] = size(128, 8192)
        c["species"] = rng.randint(1, 3)
        c["bar_w"] = round(rng.uniform(0.05, 0.2), 3)
    elif kind == "noalloc":
        c["n"] = size(64, 4096)
    else:
        c["n"] = size(64, 4096)
        c["width"] = rng.randint(160, 960)
        c["height"] = rng.randint(160, 960)
        c["images"] = c["n"] <= 200 and rng.random() < 0.5
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _full(case):
    return {**DEFAULTS, **case}


def _build(c, n, seed):
    """(spec, state) of one system of n rods: lengths around 3 with
    a spread of 0.4, random non-overlapping placement, Maxwell-Boltzmann momenta."""
    rng = np.random.default_rng([int(seed), n, 11])
    lengths = np.clip(rng.normal(3.0, 0.4, n), 2.0, 4.5)
    lengths += 3.0 - lengths.mean()  # the same volume, and so the same box, from every seed
    mu2 = 5.0 if c["field"] else MU2
    st, box = S.make_system(n=n, phi=c["phi"], lengths=lengths, mu=np.full(n, math.sqrt(mu2)),
                            seed=int(rng.integers(1 << 31)))
    if c["nd"] == 2:
        # one tilted dipole ahead of the centre and an axial one behind it
        dip = np.zeros((n, 2, 5))
        dip[:, 0] = (0.6, 0.6, 0.0, 0.8, 0.9)
        dip[:, 1] = (-0.8, 0.0, 0.0, 1.0, 0.7)
        st.dip = dip
    B = np.array([0.0, 0.0, c["field"] / math.sqrt(mu2)])
    spec = S.SystemSpec(n=n, box=box, alpha=c["alpha"] / float(box[0]), K_max=math.isqrt(c["ksq"]) + 1,
                        ksq_max=c["ksq"], dt=DT, B=B, rc_real=c["rc"], cl_energy=c["u_bond"])
    return spec, st


def _systems(c, seed):
    if c["kind"] != "batch":
        return [_build(c, c["n"], seed)]
    # N log-uniform over [n_lo, n], phi over [0.05, 0.22], the sizes the case's own
    m = c["systems"]
    q = (np.arange(m) + 1.0) / m
    ns = np.exp(math.log(c["n_lo"]) + q * math.log(c["n"] / c["n_lo"])).round().astype(int)
    subs = [dict(c, phi=0.05 + 0.17 * ((k * 0.6180339887) % 1.0)) for k in range(m)]
    order = np.argsort(-ns)
    out = [None] * len(ns)
    with ThreadPoolExecutor(8) as ex:  # the placement is host code that runs without the interpreter's lock
        for k, made in zip(order, ex.map(lambda k: _build(subs[k], int(ns[k]), 1000 * int(seed) + int(k)),
                                         order)):
            out[k] = made
    return out


def _counts(c):
    """Rods per species."""
    k = c["species"]
    first = [c["n"] // (k + 1)] * (k - 1)
    return first + [c["n"] - sum(first)]


def _host_arrays(n):
    def pin(*shape):
        return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()

    return {k: pin(n, 3, 3) if k == "O" else pin(n, 3) for k in KEYS}


def prepare(case, seed):
    c = _full(case)
    made = _systems(c, seed)
    state = {"case": c}
    if c["kind"] == "noalloc":
        spec, st = made[0]
        dev = torch.device("cuda")
        n = st.n
        state.update(
            lib=L.load(), alpha=float(spec.alpha), box=(ctypes.c_double * 3)(*[float(x) for x in spec.box]),
            pos=torch.tensor(st.r, device=dev), mom=torch.tensor(st.dip[:, 0, 4:5] * st.O[:, 2, :], device=dev),
            F=torch.empty(n, 3, dtype=torch.float64, device=dev), T=torch.empty(n, 3, dtype=torch.float64, device=dev),
            UPT=torch.empty(10, dtype=torch.float64, device=dev))
        return state
    b = L.Batch([sp for sp, _ in made], [st for _, st in made])
    state["batch"] = b
    if c["kind"] in ("host_steps", "batch"):
        n = sum(sp.n for sp, _ in made)
        state["host"] = _host_arrays(n)
        state["obs"] = (L.Observables * len(made))()
    if c["kind"] == "host_steps":
        # the forces of the first configuration, as the driver evaluates them before its loop
        b.observe()
        b.download_all(*(state["host"][k] for k in KEYS))
    if c["kind"] == "correlations":
        b.set_species(0, _counts(c))
    if c["kind"] == "picture":
        edge = float(max(made[0][0].box))
        state["view"] = L.View.make(width=c["width"], height=c["height"], theta=0.7, phi=0.4, dist=1.2 * edge,
                                    images=c["images"])
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
U_KEYS = ("U_ss", "U_dipR", "U_dipK", "U_ext", "U_self")
PT_KEYS = ("PT_kin", "PT_ss", "PT_dipR", "PT_dipK")


def _obs_arrays(buf):
    """A buffer of mdsc_observables as arrays over its systems."""
    o = np.frombuffer(buf, dtype=np.dtype(L.Observables))
    return {"U": np.stack([o[k] for k in U_KEYS], 1), "W": o["W_ss"], "K": o["K"], "xi": o["xi"],
            "PT": np.stack([o[k] for k in PT_KEYS], 1), "order": np.stack([o["G1"], o["G2"]], 1), "M": o["M"],
            "step": o["step"]}


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "noalloc":
        n = state["pos"].shape[0]
        code = state["lib"].mdsc_force_dipR_noalloc(
            n, ctypes.c_void_p(state["pos"].data_ptr()), ctypes.c_void_p(state["mom"].data_ptr()),
            ctypes.cast(state["box"], ctypes.POINTER(ctypes.c_double)), state["alpha"],
            ctypes.c_void_p(state["F"].data_ptr()), ctypes.c_void_p(state["T"].data_ptr()),
            ctypes.c_void_p(state["UPT"].data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if code != 0:
            raise L.MdscError(code, "mdsc_force_dipR_noalloc")
        return {k: state[k] for k in ("F", "T", "UPT")}
    b = state["batch"]
    if kind == "steps":
        o = b.step(c["steps"])[0]
        d = b.download(0)
        return {**{k: d[k] for k in KEYS}, "U": np.array([[o[k] for k in U_KEYS]]), "W": np.array([o["W_ss"]]),
                "K": np.array([o["K"]]), "xi": np.array([o["xi"]]), "PT": np.array([[o[k] for k in PT_KEYS]]),
                "order": np.array([[o["G1"], o["G2"]]]), "M": np.array([o["M"]]), "step": np.array([o["step"]])}
    if kind == "host_steps":
        b.step_io(state["host"], c["steps"], state["host"], state["obs"])
        return {**state["host"], **_obs_arrays(state["obs"])}
    if kind == "batch":
        b.step_io(None, c["steps"], state["host"], state["obs"])
        return {**state["host"], **_obs_arrays(state["obs"])}
    if kind == "forces":
        b.zero_forces()
        Us, W, PTs = b.force_sc()
        Ur, PTr = b.force_dipR()
        Uk, PTk = b.force_dipK()
        Ux = b.ext_field()
        U0 = b.self_ener()
        d = b.download(0)
        return {"F": d["F"], "T": d["T"], "U": np.stack([Us, Ur, Uk, Ux, U0], 1), "W": W,
                "PT": np.stack([PTs, PTr, PTk], 1).reshape(1, 3, 9)}
    if kind == "clusters":
        labels, n = b.clust_conf(0)
        return {"labels": labels, "n": n}
    if kind == "correlations":
        return {"hist": b.correlations(c["bar_w"])[0]}
    return {"rgb": b.render(0, state["view"])}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    c = _full(case)
    if c["kind"] == "batch":  # the mean of a log-uniform N, and of its square
        lo, hi = c["n_lo"], c["n"]
        lg = math.log(hi / lo)
        k = c["systems"]
        N, N2 = k * (hi - lo) / lg, k * (hi * hi - lo * lo) / (2 * lg)
    else:
        N, N2 = float(c["n"]), float(c["n"]) ** 2
    nk = 2.0 / 3.0 * math.pi * c["ksq"] ** 1.5
    pairs = 0.5 * N2 * c["nd"] ** 2
    if c["rc"]:
        vol = math.pi * 3.0 / 4 + math.pi / 6  # of a rod of length 3
        pairs = min(pairs, 0.5 * N * c["nd"] ** 2 * c["phi"] / vol * 4.0 / 3.0 * math.pi * c["rc"] ** 3)
    forces = 180.0 * pairs + 60.0 * N * c["nd"] * nk + 2000.0 * N
    state = 8.0 * 24 * N  # r, p, O, l, F, T
    shapes = 8.0 * (3 + 5 * c["nd"]) * N
    kind = c["kind"]
    if kind in ("steps", "batch", "host_steps"):
        return {"bytes": 2 * state + shapes, "flops": c["steps"] * (forces + 400.0 * N)}
    if kind == "forces":
        return {"bytes": state + shapes, "flops": forces}
    if kind == "clusters":
        return {"bytes": 8.0 * 12 * N + shapes + 4 * N, "flops": 20.0 * 150 * N}
    if kind == "correlations":
        return {"bytes": 8.0 * 6 * N, "flops": 45.0 * 0.5 * N2}
    if kind == "noalloc":
        return {"bytes": 8.0 * 12 * N, "flops": 180.0 * pairs}
    px = float(c["width"] * c["height"])
    caps = N * (27 if c["images"] else 1) * 3
    return {"bytes": 3 * px + 4 * 16 * caps, "flops": 400.0 * px + 100.0 * caps}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=_dev())


class _Exact:
    """One system in float64: the force terms and the integrator of the driver's loop."""

    def __init__(self, spec, st):
        self.n, self.nd = st.n, st.dip.shape[1]
        self.box = _t(spec.box)
        self.V = float(np.prod(spec.box))
        self.alpha, self.rc = float(spec.alpha), float(spec.rc_real)
        self.T, self.Q, self.B = float(spec.temp), float(spec.Q), _t(spec.B)
        self.r, self.p, self.O, self.l = (_t(getattr(st, k)) for k in ("r", "p", "O", "l"))
        self.len, self.dia, self.mass = _t(st.length), _t(st.dia), _t(st.mass)
        self.I = _t(S.inertia(st.length, st.dia, st.mass))
        self.off, self.body, self.mu = _t(st.dip[:, :, 0]), _t(st.dip[:, :, 1:4]), _t(st.dip[:, :, 4])
        self.xi, self.step = [float(spec.xi0)] * 2, 0
        K = spec.K_max
        g = np.arange(-(K - 1), K)
        nx, ny, nz = np.meshgrid(g, g, np.arange(K), indexing="ij")
        kn = np.stack([nx, ny, nz], -1).reshape(-1, 3)
        half = (kn[:, 2] > 0) | ((kn[:, 2] == 0) & ((kn[:, 1] > 0) | ((kn[:, 1] == 0) & (kn[:, 0] > 0))))
        kn = kn[half & ((kn ** 2).sum(1) <= spec.ksq_max if spec.ksq_max > 0 else True)]
        self.k = _t(kn) * (2 * math.pi / self.box)
        # the table of the real-space terms A, B, C the reference interpolates in
        m = torch.arange(1, 32770, dtype=torch.float64, device=_dev())
        x = LATTICE_H * m
        a2 = self.alpha ** 2
        gauss = 2 * self.alpha * torch.exp(-a2 * x * x) / math.sqrt(math.pi)
        erfc = torch.erfc(self.alpha * x)
        tab = torch.stack([erfc / x ** 3 + gauss / x ** 2,
                           (3 * erfc / x ** 3 + gauss * (2 * a2 + 3 / x ** 2)) / x ** 2, 4 * a2 * a2 * gauss], 1)
        if self.rc > 0:
            tab[x > self.rc] = 0.0
        self.tab = tab
        self.forces()

    def mimg(self, d):
        return d - self.box * torch.floor(d / self.box + 0.5)

    def dipoles(self):
        """Positions and moments of every dipole, and its rod."""
        pos = self.r[:, None, :] + self.off[..., None] * self.O[:, None, 2, :]
        m = self.mu[..., None] * torch.einsum("nba,nwb->nwa", self.O, self.body)
        owner = torch.arange(self.n, device=_dev())[:, None].expand(self.n, self.nd)
        return pos.reshape(-1, 3), m.reshape(-1, 3), owner.reshape(-1)

    def real(self, pos, m, owner):
        N = len(pos)
        F, E = torch.zeros_like(pos), torch.zeros_like(pos)
        U, PT = 0.0, torch.zeros(3, 3, dtype=torch.float64, device=_dev())
        rows = max(1, min(N, (1 << 24) // N))
        for i0 in range(0, N, rows):
            mi = m[i0:i0 + rows]
            d = [pos[i0:i0 + rows, a, None] - pos[None, :, a] for a in range(3)]
            d = [x - self.box[a] * torch.floor(x / self.box[a] + 0.5) for a, x in enumerate(d)]
            on = owner[i0:i0 + rows, None] != owner[None, :]
            r2 = torch.where(on, d[0] * d[0] + d[1] * d[1] + d[2] * d[2], 1.0)
            q = torch.sqrt(r2) / LATTICE_H
            idx = torch.floor(q).long().clamp(1, 32767)
            fr = q - idx
            lo, hi = self.tab[idx - 1], self.tab[idx]
            A, Bt, C = [(lo[..., k] + fr * (hi[..., k] - lo[..., k])) * on for k in range(3)]
            del lo, hi, idx, fr, q
            mimj = mi @ m.T
            mir = sum(mi[:, a, None] * d[a] for a in range(3))
            mjr = sum(m[None, :, a] * d[a] for a in range(3))
            qq = mir * mjr / r2
            U += float((mimj * A - mir * mjr * Bt).sum()) / 2
            fact = (mimj - 5 * qq) * Bt - qq * C
            for a in range(3):
                f = fact * d[a] + Bt * (mir * m[None, :, a] + mjr * mi[:, a, None])
                F[i0:i0 + rows, a] = f.sum(1)
                E[i0:i0 + rows, a] = (mjr * Bt * d[a] - A * m[None, :, a]).sum(1)
                for c in range(3):
                    PT[c, a] += (d[c] * f).sum() / 2
        return F, torch.linalg.cross(m, E), U, PT

    def recip(self, pos, m):
        k = self.k
        k2 = (k * k).sum(1)
        val = 8 * math.pi * torch.exp(-k2 / (4 * self.alpha ** 2)) / k2 / self.V
        ph = pos @ k.T
        e = torch.complex(torch.cos(ph), -torch.sin(ph))  # exp(-i k.r) of every dipole
        del ph
        a = m @ k.T
        s = a * e
        nd = self.nd
        Si = s.reshape(self.n, nd, -1).sum(1)
        Ui = [(m[:, c, None] * e).reshape(self.n, nd, -1).sum(1) for c in range(3)]
        Sk, Uk = Si.sum(0), [u.sum(0) for u in Ui]
        nrm = Sk.abs() ** 2 - (Si.abs() ** 2).sum(0)
        U = float((val * nrm / 2).sum())
        pval = 2 * (1 / (4 * self.alpha) + 1 / k2)
        PT = torch.zeros(3, 3, dtype=torch.float64, device=_dev())
        for j in range(3):
            re = (Sk.conj() * Uk[j]).real - (Si.conj() * Ui[j]).real.sum(0)
            for q in range(3):
                t = ((1.0 if j == q else 0.0) - pval * k[:, j] * k[:, q]) * nrm + 2 * re * k[:, q]
                PT[j, q] = (val * t / 2).sum()
        D = (val * Sk).conj()[None, :] - val * Si.conj()
        Z = e * D.repeat_interleave(nd, 0)
        return (-a * Z.imag) @ k, torch.linalg.cross(m, -Z.real @ k), U, PT

    def wca(self):
        n = self.n
        F, T = torch.zeros_like(self.r), torch.zeros_like(self.r)
        reach = float(self.len.max() + 1.13 * self.dia.max())
        pi, pj = [], []
        rows = max(1, min(n, (1 << 24) // n))
        for i0 in range(0, n, rows):
            d2 = 0
            for a in range(3):
                x = self.r[i0:i0 + rows, a, None] - self.r[None, :, a]
                x = x - self.box[a] * torch.floor(x / self.box[a] + 0.5)
                d2 = d2 + x * x
            i, j = torch.nonzero(d2 < reach * reach, as_tuple=True)
            i = i + i0
            keep = i < j
            pi.append(i[keep])
            pj.append(j[keep])
        i, j = torch.cat(pi), torch.cat(pj)
        rij = self.mimg(self.r[i] - self.r[j])
        di, dj = self.len[i, None] * self.O[i, 2], self.len[j, None] * self.O[j, 2]
        # closest points of the segments w + s di - t dj, s and t in [0, 1]
        w = rij - 0.5 * di + 0.5 * dj
        a, e, bb = (di * di).sum(1), (dj * dj).sum(1), (di * dj).sum(1)
        cc, f = (di * w).sum(1), (dj * w).sum(1)
        den = a * e - bb * bb
        s = torch.where(den > 1e-12, ((bb * f - cc * e) / den.clamp_min(1e-12)).clamp(0, 1), 0.0)
        t = (bb * s + f) / e
        s = torch.where(t < 0, (-cc / a).clamp(0, 1), torch.where(t > 1, ((bb - cc) / a).clamp(0, 1), s))
        t = t.clamp(0, 1)
        dij = w + s[:, None] * di - t[:, None] * dj
        dsq = (dij * dij).sum(1)
        sig2 = ((self.dia[i] + self.dia[j]) / 2) ** 2
        on = dsq < 2.0 ** (1.0 / 3.0) * sig2
        i, j, rij, dij, dsq, sig2 = i[on], j[on], rij[on], dij[on], dsq[on], sig2[on]
        s, t, di, dj = s[on], t[on], di[on], dj[on]
        s6 = (sig2 / dsq) ** 3
        f = (24 * (2 * s6 * s6 - s6) / dsq)[:, None] * dij
        F.index_add_(0, i, f)
        F.index_add_(0, j, -f)
        T.index_add_(0, i, torch.linalg.cross((s - 0.5)[:, None] * di, f))
        T.index_add_(0, j, torch.linalg.cross((t - 0.5)[:, None] * dj, -f))
        return F, T, float((4 * (s6 * s6 - s6) + 1).sum()), float((rij * f).sum()), rij.T @ f

    def self_energy(self):
        U = 0.0
        for v in range(self.nd):
            for w in range(v + 1, self.nd):
                z = self.off[:, v] - self.off[:, w]
                uv = (self.body[:, v] * self.body[:, w]).sum(1)
                zz = self.body[:, v, 2] * self.body[:, w, 2]
                U += float((self.mu[:, v] * self.mu[:, w] * (uv - 3 * zz) / z.abs() ** 3).sum())
        return U

    def forces(self):
        pos, m, owner = self.dipoles()
        self.F, self.Tq, Us, self.W, PTs = self.wca()
        Fr, Tr, Ur, PTr = self.real(pos, m, owner)
        Fk, Tk, Uk, PTk = self.recip(pos, m)
        f = Fr + Fk
        t = Tr + Tk + torch.linalg.cross(m, self.B.expand_as(m))
        arm = (self.off[..., None] * self.O[:, None, 2, :]).reshape(-1, 3)
        t = t + torch.linalg.cross(arm, f)
        self.F = self.F + f.reshape(self.n, self.nd, 3).sum(1)
        self.Tq = self.Tq + t.reshape(self.n, self.nd, 3).sum(1)
        self.U = [Us, Ur, Uk, -float((m @ self.B).sum()), self.self_energy()]
        self.PT = [PTs, PTr, PTk]

    def kinetic(self):
        lb = torch.einsum("nab,nb->na", self.O, self.l)
        return float((self.p ** 2).sum(1).div(self.mass).sum()) / 2, float((lb ** 2 / self.I).sum()) / 2

    def renorm(self):
        u = self.O[:, 2] / self.O[:, 2].norm(dim=1, keepdim=True)
        v = u + self.O[:, 1]
        v = v - (v * u).sum(1, keepdim=True) * u
        v = v / v.norm(dim=1, keepdim=True)
        self.O = torch.stack([torch.linalg.cross(v, u), v, u], 1)

    def rotate(self):
        O = self.O.clone()
        for axis, part in ((0, 0.5), (1, 0.5), (2, 1.0), (1, 0.5), (0, 0.5)):
            lb = torch.einsum("nab,nb->na", O, self.l)
            a = -lb[:, axis] * part * DT / self.I[:, axis]
            i, j = (axis + 1) % 3, (axis + 2) % 3
            ca, sa = torch.cos(a)[:, None], torch.sin(a)[:, None]
            O[:, i], O[:, j] = ca * O[:, i] - sa * O[:, j], sa * O[:, i] + ca * O[:, j]
        self.O = O

    def advance(self, steps):
        h = 0.5 * DT
        for _ in range(steps):
            if self.step % 100 == 0:
                self.renorm()
            self.p = (self.p + h * self.F) / (1 + h * self.xi[0])
            self.l = (self.l + h * self.Tq) / (1 + h * self.xi[1])
            self.xi = [x + DT * (2 * K - 3 * self.n * self.T) / self.Q for x, K in zip(self.xi, self.kinetic())]
            self.r = self.r + DT * self.p / self.mass[:, None]
            self.rotate()
            self.forces()
            self.p = self.p * (1 - h * self.xi[0]) + h * self.F
            self.l = self.l * (1 - h * self.xi[1]) + h * self.Tq
            self.step += 1

    def observables(self):
        u = self.O[:, 2]
        Q = (3 * u.T @ u - self.n * torch.eye(3, dtype=torch.float64, device=_dev())) / (2 * self.n)
        ev, vec = np.linalg.eigh(Q.cpu().numpy())
        k = int(np.argmax(np.abs(ev)))
        G1 = abs(float(u.sum(0).cpu().numpy() @ vec[:, k])) / self.n
        PT = [torch.einsum("na,nc,n->ac", self.p, self.p, 1 / self.mass)] + self.PT
        return {"U": self.U, "W": self.W, "K": self.kinetic(), "xi": self.xi,
                "PT": [x.reshape(-1).tolist() for x in PT], "order": [G1, abs(float(ev[k]))],
                "M": self.dipoles()[1].sum(0).tolist()}

    def state(self):
        return {"r": self.r, "p": self.p, "O": self.O, "l": self.l, "F": self.F, "T": self.Tq}


def _exact_correlations(c, spec, st):
    r, u, box = _t(st.r), _t(st.O[:, 2]), _t(spec.box)
    n, w = st.n, c["bar_w"]
    counts = _counts(c)
    nc = len(counts)
    nb = int(math.floor(math.sqrt(3.0) * float(min(spec.box)) / (2.0 * w)))
    sp = torch.repeat_interleave(torch.arange(nc, device=_dev()), torch.tensor(counts, device=_dev()))
    blocks = nc + nc * (nc - 1) // 2
    hist = torch.zeros(4, blocks * nb, dtype=torch.float64, device=_dev())
    rows = max(1, min(n, (1 << 23) // n))
    for i0 in range(0, n, rows):
        d = r[i0:i0 + rows, None, :] - r[None]
        d = d - box * torch.floor(d / box + 0.5)
        R = d.norm(dim=-1)
        i = torch.arange(i0, min(n, i0 + rows), device=_dev())
        b = torch.floor(R / w).long()
        on = (i[:, None] < torch.arange(n, device=_dev())[None, :]) & (b < nb)
        a, q = torch.nonzero(on, as_tuple=True)
        d, R, b = d[on], R[on], b[on]
        ui, uj, si, sj = u[i0 + a], u[q], sp[i0 + a], sp[q]
        dot = (ui * uj).sum(1)
        dd = (ui * d).sum(1) * (uj * d).sum(1) / R ** 2
        blk = torch.where(si == sj, si, nc + si * (2 * nc - si - 1) // 2 + (sj - si - 1))
        f = torch.where(si == sj, 2.0, 1.0)
        for k, v in enumerate((f, f * dot, f * (3 * dd - dot), 0.5 * f * (3 * dot * dot - 1))):
            hist[k] += torch.bincount(blk * nb + b, weights=v, minlength=blocks * nb)
    return hist.reshape(4, blocks, nb).permute(1, 0, 2).contiguous()


def exact(case, seed):
    c = _full(case)
    kind = c["kind"]
    if kind in ("clusters", "picture"):
        return None  # labels and pixels: whole numbers
    made = _systems(c, seed)
    if kind == "correlations":
        return {"hist": _exact_correlations(c, *made[0])}
    if kind == "noalloc":
        x = _Exact(*made[0])
        F, T, U, PT = x.real(*x.dipoles())
        return {"F": F, "T": T, "UPT": torch.cat([_t([U]), PT.reshape(-1)])}
    xs = [_Exact(*m) for m in made]
    if kind == "forces":
        x = xs[0]
        return {"F": x.F, "T": x.Tq, "U": np.array([x.U]), "W": np.array([x.W]),
                "PT": torch.stack(x.PT).reshape(1, 3, 9)}
    for x in xs:
        x.advance(c["steps"])
    out = {k: torch.cat([x.state()[k] for x in xs]) for k in KEYS}
    obs = [x.observables() for x in xs]
    out.update({k: np.array([o[k] for o in obs]) for k in ("U", "W", "K", "xi", "PT", "order", "M")})
    out["step"] = None
    return out
