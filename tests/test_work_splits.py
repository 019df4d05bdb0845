"""The splits of a step's work that a small batch runs on (one k tile per
gather block, one k-vector per structure-factor thread) and those of a batch
that fills the GPU give a system the same bits, at the edges of their blocks
and tiles; and both agree with the oracle."""
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
         (130, 4, 9)]


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
