"""The geometric cluster criterion where the reference's segment distance is not
the smallest one, or not a clear one (spherocyl_dist, v25/functions.cpp:89-489):
axis lines that meet (an end point's distance to the other segment), nearly
parallel axes, and rods of no or little length.

The bond of a pair is the oracle's distance of the lower index to the higher
against (D + min_s)^2: where axis lines meet, the routine's distance can depend
on the order of the two, and the reference asks in the order of its draws.  Where
it does not, the labels are the oracle's.
"""
import numpy as np
import pytest

import hand_configs as H
import oracle
from mdspherocyl_gb300 import lib as L
from mdspherocyl_gb300 import systems as S

MIN_S = 0.25
THR = (1.0 + MIN_S) ** 2
CELL = 12.0  # a pair to a cell of this edge
SIDE = 6     # cells along the box


def _pair(kind, rng):
    """One pair whose bond is in question: relative positions, axes, lengths."""
    la, lb = rng.uniform(0.5, 4.0, 2)
    a = rng.uniform(0, 2 * np.pi)
    b = a + 10.0 ** rng.uniform(-7, -0.5) if kind == "nearly-parallel" else rng.uniform(0, 2 * np.pi)
    oa, ob = (np.array([np.cos(x), np.sin(x), 0.0]) for x in (a, b))
    # a point of each rod's axis, 0.3 to 1.6 apart in the plane
    g = rng.uniform(0, 2 * np.pi)
    w = rng.uniform(0.3, 1.6) * np.array([np.cos(g), np.sin(g), 0.0])
    rb = rng.uniform(-0.5, 0.5) * la * oa + w - rng.uniform(-0.5, 0.5) * lb * ob
    if kind == "near-crossing":  # out of the plane by little: on both sides of 1e-6
        rb[2] = 10.0 ** rng.uniform(-8, -1)
    if kind == "nearly-parallel" and rng.uniform() < 0.5:
        rb[2] = rng.uniform(0.0, 1.3)
    if kind == "short":  # the first rod without length, or nearly
        la = 0.0 if rng.uniform() < 0.5 else 10.0 ** rng.uniform(-4, -1)
        rb = rng.uniform(-0.6, 0.6) * lb * ob + rng.uniform(0.3, 1.6) * np.array([np.cos(g), 0.0, np.sin(g)])
    q = H._rotation(rng, False)
    return np.array([[0.0, 0.0, 0.0], q @ rb]), (q @ oa, q @ ob), (la, lb)


def _system(pairs):
    box = np.full(3, CELL * SIDE)
    anchors = (np.array(np.unravel_index(np.arange(len(pairs)), (SIDE,) * 3)).T + 0.5) * CELL
    anchors = anchors + np.array([0.0, 0.0, 0.5 * CELL])  # the last layer crosses the face
    r = np.mod(np.concatenate([c + rel for c, (rel, _, _) in zip(anchors, pairs)]), box)
    O = np.array([H.frame(o / np.sqrt(o @ o)) for _, ax, _ in pairs for o in ax])
    ln = np.array([x for _, _, lens in pairs for x in lens])
    n = len(ln)
    st = S.SystemState(r, np.zeros((n, 3)), O, np.zeros((n, 3)), ln, np.ones(n), np.ones(n), np.zeros((n, 1, 5)))
    return S.SystemSpec(n=n, box=box, alpha=6.0 / box[0], K_max=2, ksq_max=1, min_s=MIN_S), st


def _osys(spec, st):
    return oracle.System(st.r, st.p, st.O, st.l, st.length, st.dia, st.mass, st.dip, spec.box)


def _bonds(orc, spec, st):
    """The routine's answer for every pair, in both orders."""
    o, n = _osys(spec, st), len(st.length)
    ask = lambda i, j: orc.seg_dist(o, i, j)[0] < THR  # noqa: E731
    return (np.array([ask(k, k + 1) for k in range(0, n, 2)]), np.array([ask(k + 1, k) for k in range(0, n, 2)]))


def _smallest(spec, st):
    """The smallest distance squared of every pair of the axis segments: from
    points along the first to the second."""
    A, B = slice(0, None, 2), slice(1, None, 2)
    r = st.r[A] - st.r[B]
    r = r - spec.box * np.floor(r / spec.box + 0.5)
    s = np.linspace(-0.5, 0.5, 401)[None, :, None]
    p = r[:, None] + s * (st.length[A, None] * st.O[A, 2])[:, None]
    t = np.clip(np.einsum("kqc,kc->kq", p, st.O[B, 2]), -st.length[B, None] / 2, st.length[B, None] / 2)
    v = p - t[:, :, None] * st.O[B, 2][:, None]
    return np.einsum("kqc,kqc->kq", v, v).min(axis=1)


def _systems(orc, kind, count, seed):
    """`count` systems of 216 pairs; of the coplanar ones every second system only
    pairs nearer than the threshold by their smallest distance and beyond it by
    the routine's."""
    rng = np.random.default_rng(seed)
    out = []
    while len(out) < count:
        pairs = []
        while len(pairs) < SIDE ** 3:
            new = [_pair(kind, rng) for _ in range(SIDE ** 3)]
            if kind == "coplanar" and len(out) % 2:
                spec, st = _system(new)
                keep = (_smallest(spec, st) < THR) & ~_bonds(orc, spec, st)[0]
                new = [p for p, k in zip(new, keep) if k]
            pairs += new
        out.append(_system(pairs[:SIDE ** 3]))
    return out


# two coplanar pairs within the threshold by their smallest distance (1.05, 1.32)
# and beyond it by the routine's
EXAMPLES = [
    (np.array([[0.0, 0.0, 0.0], [-2.25, 0.75, 0.0]]),
     (np.array([1.0, 0.0, 0.0]), np.array([np.cos(np.pi / 6), np.sin(np.pi / 6), 0.0])), (3.0, 3.0), 2.25),
    (np.array([[0.0, 0.0, 0.0], [1.94240274, -1.29608309, 0.0]]),
     (np.array([-0.65793464, 0.75307503, 0.0]), np.array([-0.16332941, 0.98657159, 0.0])),
     (2.117187924736352, 3.718218768764231), 2.522),
]


def test_the_routine_is_not_the_smallest_distance(orc):
    spec, st = _system([e[:3] for e in EXAMPLES])
    assert np.all(_smallest(spec, st) < 0.9 * THR)
    for k, e in enumerate(EXAMPLES):
        assert abs(orc.seg_dist(_osys(spec, st), 2 * k, 2 * k + 1)[0] - e[3]) < 1e-3


@pytest.mark.gpu
def test_examples_are_not_bonded():
    spec, st = _system([e[:3] for e in EXAMPLES])
    with L.Batch([spec], [st]) as bt:
        lab, nc = bt.clust_conf(0)
    assert nc == 4 and len(set(lab)) == 4


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["coplanar", "near-crossing", "nearly-parallel", "short"])
def test_bonds_of_pairs_equal_the_oracle(orc, kind):
    systems = _systems(orc, kind, 6, 50)
    with L.Batch([s for s, _ in systems], [t for _, t in systems]) as bt:
        for k, (spec, st) in enumerate(systems):
            lab, nc = bt.clust_conf(k)
            lower, higher = _bonds(orc, spec, st)
            bonded = lab[0::2] == lab[1::2]
            assert np.array_equal(bonded, lower), (kind, k, np.flatnonzero(bonded != lower))
            assert nc == 2 * len(lower) - lower.sum()
            if np.array_equal(lower, higher):
                want, nw, _ = orc.clust_conf(_osys(spec, st), MIN_S)
                assert nc == nw and np.array_equal(lab, want)
