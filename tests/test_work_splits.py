"""How work is split over the GPU, at the edges of the splits.

The splits of a step that a small batch runs on (one k tile per gather block,
one k-vector per structure-factor thread) and those of a batch that fills the
GPU give a system the same bits, and both agree with the oracle; so do the
clusters, histograms and pictures.
"""
import ctypes
import math

import numpy as np
import pytest

import oracle
from conftest import rms_rel
from mdspherocyl_gb300 import lib as L
from mdspherocyl_gb300 import systems as S

pytestmark = pytest.mark.gpu

TOL_F = 1e-5  # the bar of the Ewald forces

# rods, dipoles per rod, |n|^2 limit: one particle block and its edges, one
# k tile (13, 62 and 128 k-vectors) and several, chunks of 256 rods and one more
SIZES = [(2, 1, 3), (64, 1, 9), (128, 1, 16), (129, 1, 36), (257, 1, 64), (700, 1, 27), (65, 2, 27), (257, 2, 36),
         (130, 4, 9), (1030, 3, 27)]


def _system(n, nd, ksq, seed):
    st, box = S.make_system(n=n, phi=0.06, lengths=np.full(n, 3.0), mu=np.full(n, 1.2), seed=seed)
    if nd > 1:
        dip = np.zeros((n, nd, 5))
        for w in range(nd):
            dip[:, w] = (0.5 * w - 0.7, 0.6, 0.0, 0.8, 0.5 + 0.2 * w)
        st.dip = dip
    spec = S.SystemSpec(n=n, box=box, alpha=6.0 / float(box[0]), K_max=math.isqrt(ksq) + 1, ksq_max=ksq,
                        B=np.array([0.1, -0.2, 0.3]))
    return spec, st


@pytest.fixture(scope="module")
def systems():
    return [_system(n, nd, ksq, 900 + k) for k, (n, nd, ksq) in enumerate(SIZES)]


@pytest.fixture(scope="module")
def in_full_batch(systems):
    """Observables and states of three steps beside 320 filler systems."""
    fill = _system(128, 1, 27, 5)
    everyone = systems + [fill] * 320
    with L.Batch([s for s, _ in everyone], [t for _, t in everyone]) as bt:
        obs = bt.step(3)
        return [(obs[k], bt.download(k)) for k in range(len(systems))]


@pytest.mark.parametrize("k", range(len(SIZES)), ids=["n%d_nd%d_k%d" % s for s in SIZES])
def test_same_bits_alone_and_in_a_full_batch(systems, in_full_batch, k):
    spec, st = systems[k]
    with L.Batch([spec], [st]) as bt:
        obs, d = bt.step(3)[0], bt.download(0)
    obs_b, d_b = in_full_batch[k]
    for f in ("r", "p", "O", "l", "F", "T"):
        assert np.array_equal(d[f], d_b[f]), f
    for key in ("U_ss", "U_dipR", "U_dipK", "U_ext", "K", "PT_dipR", "PT_dipK", "PT_kin", "PT_ss", "xi", "G1", "G2",
                "M"):
        assert np.array_equal(np.asarray(obs[key]), np.asarray(obs_b[key])), key


@pytest.mark.parametrize("k", range(len(SIZES)), ids=["n%d_nd%d_k%d" % s for s in SIZES])
def test_forces_against_the_oracle(systems, k):
    spec, st = systems[k]
    orc = oracle.Oracle()
    with L.Batch([spec], [st]) as bt:
        for name, call in (("dipK", lambda o: orc.force_dipK(o, spec.K_max, spec.alpha, spec.ksq_max)),
                           ("dipR", lambda o: orc.force_dipR(o, spec.alpha))):
            bt.zero_forces()
            U, PT = getattr(bt, "force_" + name)()
            d = bt.download(0)
            o = oracle.System(st.r, st.p, st.O, st.l, st.length, st.dia, st.mass, st.dip, spec.box)
            Uo, PTo = call(o)
            assert rms_rel(d["F"], o.F) <= TOL_F, name
            assert rms_rel(d["T"], o.T) <= TOL_F, name
            assert rms_rel(PT[0], PTo) <= TOL_F, name
            assert abs(U[0] - Uo) <= TOL_F * max(abs(Uo), np.abs(PTo).max()), name


# ---- strips of 64 dipoles: a lone one, one dipole in the last, as many as the
# force assembly adds by itself (32) and one more -----------------------------
@pytest.mark.parametrize("n", [2, 64, 65, 2048, 2049])
def test_real_space_strips_against_the_oracle(n):
    """The batch's own sums over the strips and those of the call that holds no
    GPU memory of its own."""
    import torch

    spec, st = _plain(n, 300 + n)
    o = _osys(spec, st)
    Uo, PTo = oracle.Oracle().force_dipR(o, spec.alpha)
    with L.Batch([spec], [st]) as bt:
        bt.zero_forces()
        U, PT = bt.force_dipR()
        d = bt.download(0)
    pos, mom = (torch.tensor(x, dtype=torch.float64, device="cuda:0")
                for x in (st.r, st.dip[:, 0, 4:5] * st.O[:, 2, :]))
    F, T, UPT = (torch.zeros(k, dtype=torch.float64, device="cuda:0") for k in ((n, 3), (n, 3), (10,)))
    box = (ctypes.c_double * 3)(*[float(x) for x in spec.box])
    code = L.load().mdsc_force_dipR_noalloc(
        n, *(ctypes.c_void_p(x.data_ptr()) for x in (pos, mom)), ctypes.cast(box, ctypes.POINTER(ctypes.c_double)),
        float(spec.alpha), *(ctypes.c_void_p(x.data_ptr()) for x in (F, T, UPT)),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert code == 0
    upt = UPT.cpu().numpy()
    for f, t, u, pt in ((d["F"], d["T"], U[0], PT[0]), (F.cpu().numpy(), T.cpu().numpy(), upt[0], upt[1:].reshape(3, 3))):
        assert rms_rel(f, o.F) <= TOL_F
        assert rms_rel(t, o.T) <= TOL_F
        assert rms_rel(pt, PTo) <= TOL_F
        assert abs(u - Uo) <= TOL_F * max(abs(Uo), np.abs(PTo).max())


# ---- clusters, histograms and pictures at the edges of their splits --------
def _plain(n, seed, phi=0.1, mu=2.2):
    rng = np.random.default_rng(seed)
    st, box = S.make_system(n=n, phi=phi, lengths=rng.uniform(2.0, 4.0, n), mu=np.full(n, mu), seed=seed)
    spec = S.SystemSpec(n=n, box=box, alpha=6.0 / float(box[0]), K_max=2, ksq_max=1)
    return spec, st


def _osys(spec, st):
    return oracle.System(st.r, st.p, st.O, st.l, st.length, st.dia, st.mass, st.dip, spec.box)


@pytest.mark.parametrize("n,u_bond", [(2, 1.0), (32, 0.0), (129, 0.8), (700, 0.0), (700, 0.8), (4095, 0.8),
                                      (4500, 0.0), (4500, 0.8)])
def test_cluster_labels_equal_the_oracle(n, u_bond):
    """Geometric and energy bonds; systems below 4096 rods screen all pairs,
    the others the cells around each rod; three calls, the second and third
    on the list the first one built."""
    spec, st = _plain(n, 60 + n, phi=0.2)
    spec.min_s, spec.cl_energy = 0.25, u_bond
    orc = oracle.Oracle()
    skip = 0
    with L.Batch([spec], [st]) as bt:
        for _ in range(3):
            lab, nc = bt.clust_conf(0)
            o = _osys(spec, st)
            want, nw, _ = (orc.clust_energy(o, u_bond * spec.temp, skip=skip) if u_bond
                           else orc.clust_conf(o, spec.min_s, skip=skip))
            assert nc == nw
            assert np.array_equal(lab, want)
            skip += nw  # one draw per cluster


@pytest.mark.parametrize("n,counts,bar_w", [(1, [1], 0.2), (128, [128], 0.1), (129, [1, 128], 0.1),
                                            (700, [128, 256, 316], 0.05), (1300, [650, 650], 0.002),
                                            (1300, [1300], 0.1)])
def test_histograms_equal_the_oracle(n, counts, bar_w):
    """Tile edges, several tiles between flushes, and (bar_w = 0.002) more bins
    than shared memory holds: counts equal, the others to the FP32 of a pair's
    term, as in the observables' tests."""
    spec, st = _plain(n, 90 + n)
    orc = oracle.Oracle()
    with L.Batch([spec], [st]) as bt:
        bt.set_species(0, counts)
        got = bt.correlations(bar_w)[0]
    want = orc.acc_correl_species(_osys(spec, st), counts, bar_w, got.shape[2])
    for q in range(want.shape[0]):
        assert np.array_equal(got[q][0], want[q][0]), q
        pairs = want[q][0] / (2.0 if q < len(counts) else 1.0)
        assert np.all(np.abs(got[q][1:] - want[q][1:]) <= 5e-6 * pairs + 1e-7), q


@pytest.mark.parametrize("n,width,height,dist", [(3, 16, 8, 8.0), (60, 77, 41, 14.0), (300, 96, 65, 3.0)])
def test_picture_close_to_the_restatement(n, width, height, dist):
    """Sizes that are no multiple of a block of pixels, and a camera inside the
    box: as the picture's tests, all but 2% of the pixels within 3 levels."""
    from oracle import render_np

    spec, st = _plain(n, 30 + n, phi=0.05)
    with L.Batch([spec], [st]) as bt:
        img = bt.render(0, width=width, height=height, theta=0.8, phi=0.3, dist=dist)
    want = render_np.render(width, height, st.r, st.O, st.length, st.dia, np.zeros(n, int), st.dip, spec.box,
                            theta=0.8, phi=0.3, dist=dist)
    off = np.abs(img.astype(int) - want.astype(int)).max(axis=-1) > 3
    assert off.mean() <= 0.02, off.mean()


@pytest.mark.parametrize("n,steps", [(2, 1), (129, 16), (129, 17), (8192, 1), (8193, 1)])
def test_step_io_from_pinned_and_pageable_arrays(n, steps):
    """State arrays the device reads and writes by itself (pinned, up to 8192
    rods) and by copies, noise with the launch (up to 16 steps) and by a copy:
    the same bits as a call on pageable arrays and as steps without them."""
    import torch

    spec, st = _plain(n, 700 + n)
    width = {"r": 3, "p": 3, "O": 9, "l": 3, "F": 3, "T": 3}
    with L.Batch([spec], [st]) as bt:
        bt.step(1)
        first = bt.download(0)
        bt.step(steps)
        bt.step(steps)
        want = bt.download(0)
    for pin in (True, False):
        host = {k: (torch.empty(n, w, dtype=torch.float64, pin_memory=pin).numpy()) for k, w in width.items()}
        with L.Batch([spec], [st]) as bt:
            bt.step(1)
            for k in host:
                host[k][...] = np.asarray(first[k]).reshape(n, width[k])
            obs = (L.Observables * 1)()
            for _ in range(2):
                bt.step_io(host, steps, host, obs)
            assert obs[0].step == 1 + 2 * steps
        for k in host:
            assert np.array_equal(host[k], np.asarray(want[k]).reshape(n, width[k])), (pin, k)


@pytest.mark.parametrize("n", [1, 2048, 2049, 9000])
def test_downloads_into_any_host_memory(n):
    """Through the batch's own pinned memory (up to 2048 rods) or straight into
    plain arrays, new or in use, and into pinned ones: the same state."""
    import torch

    spec, st = _plain(n, 40 + n)
    width = (3, 3, 9, 3, 3, 3)
    with L.Batch([spec], [st]) as bt:
        bt.observe()
        d = bt.download(0)
        want = [np.asarray(d[k]).reshape(n, w) for k, w in zip(("r", "p", "O", "l", "F", "T"), width)]
        assert np.array_equal(want[0], st.r) and np.abs(want[4]).max() < np.inf
        pinned = [torch.full((n, w), 7.0, dtype=torch.float64, pin_memory=True).numpy() for w in width]
        mixed = [np.full((n, w), 7.0) if k % 2 else x.copy() * 0 for k, (w, x) in enumerate(zip(width, pinned))]
        for arrays in (pinned, mixed, mixed, pinned[:2] + mixed[2:]):
            bt.download_all(*arrays)
            for got, x in zip(arrays, want):
                assert np.array_equal(got, x)


@pytest.mark.parametrize("steps", [3, 4, 5, 8])
def test_steps_in_pairs_and_one_by_one(steps):
    """A call of several steps runs two to a graph; a step limit inside a pair and
    a trace of every step (one to a graph) leave the same states."""
    spec, st = _plain(130, 77)
    with L.Batch([spec], [st]) as bt:
        for _ in range(steps):
            one = bt.step(1)[0]
        want = bt.download(0)
    with L.Batch([spec, spec], [st, st]) as bt:
        bt.set_step_limit(1, steps - 2)
        obs = bt.step(steps)
        got, short = bt.download(0), bt.download(1)
    with L.Batch([spec], [st]) as bt:
        bt.step(steps - 2)
        before = bt.download(0)
    assert obs[0]["step"] == one["step"] == steps and obs[1]["step"] == steps - 2
    for k in ("r", "p", "O", "l", "F", "T"):
        assert np.array_equal(got[k], want[k]), k
        assert np.array_equal(short[k], before[k]), k
