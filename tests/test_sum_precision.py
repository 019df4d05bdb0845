"""Sums to FP64's accuracy: partial results of very different size that cancel are
no further from the exact sum than an FP64 sum of them, and a sum that is not a
number stays none.

The inputs put one exactly known term into each partial sum: five of them, big +
middle + tiny - big - middle with 24 bits each from 1 down to about 2^-51, which
53 bits hold.
"""
import ctypes
import math
from fractions import Fraction

import numpy as np
import pytest

from mdspherocyl_gb300 import lib as L
from mdspherocyl_gb300 import systems as S

pytestmark = pytest.mark.gpu

BIG, MIDDLE, TINY = 1.0, 1.2345678 * 2.0 ** -14, 1.3571113 * 2.0 ** -27
BOX = 64.0  # positions on multiples of 2^-20: exact in the box's fixed point


def _noalloc(pos, mom, alpha):
    import torch

    n = len(pos)
    x, m = (torch.tensor(a, dtype=torch.float64, device="cuda:0") for a in (pos, mom))
    F, T, UPT = (torch.full(k, 7.0, dtype=torch.float64, device="cuda:0") for k in ((n, 3), (n, 3), (10,)))
    box = (ctypes.c_double * 3)(BOX, BOX, BOX)
    code = L.load().mdsc_force_dipR_noalloc(
        n, *(ctypes.c_void_p(a.data_ptr()) for a in (x, m)), ctypes.cast(box, ctypes.POINTER(ctypes.c_double)),
        float(alpha), *(ctypes.c_void_p(a.data_ptr()) for a in (F, T, UPT)),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert code == 0
    return F.cpu().numpy(), T.cpu().numpy(), UPT.cpu().numpy()


def _grid(n):
    """n places of a coarse grid, none of them near the box's centre."""
    k = np.arange(n)
    return np.stack([k % 16, k // 16 % 16, 4.0 * (k // 256)], axis=1) * np.array([4.0, 4.0, 1.0]) + 1.0


@pytest.mark.parametrize("sign,what", [(1.0, "force"), (-1.0, "torque")])
def test_noalloc_adds_a_dipoles_strips_in_fp64(sign, what):
    """One partner of dipole 0 in each of five strips, the last two mirror images
    of the first two: with the same moment their force is the opposite one, with
    the opposite moment their torque."""
    n = 64 * 6
    centre = np.full(3, BOX / 2)
    at = [np.array([1.5, 0.25, -0.5]), np.array([0.25, 1.75, 0.5]), np.array([-0.5, 0.75, 1.5])]
    at += [-at[0], -at[1]]
    size = [BIG, MIDDLE, TINY, sign * BIG, sign * MIDDLE]

    def run(which):
        pos, mom = _grid(n), np.zeros((n, 3))
        pos[0], mom[0] = centre, (0.375, 0.75, -0.625)
        for k in range(5):
            pos[64 * (k + 1)] = centre + at[k]
            if k in which:
                mom[64 * (k + 1)] = size[k] * np.array([0.5, -0.875, 0.75])
        F, T, _ = _noalloc(pos, mom, 0.5)
        return (F if what == "force" else T)[0]

    term = [run([k]) for k in range(5)]
    assert np.array_equal(term[3], -term[0]) and np.array_equal(term[4], -term[1])
    assert np.all(term[2] != 0)
    got = run(range(5))
    for c in range(3):
        exact = math.fsum(t[c] for t in term)
        fp64 = 0.0
        for t in term:  # strip by strip
            fp64 += t[c]
        assert abs(got[c] - exact) <= abs(fp64 - exact), (c, got[c], fp64, exact)


def test_noalloc_adds_the_tiles_in_fp64():
    """Five pairs, each in a tile of its own and beyond reach of the others: the
    energies and pressure terms of two cancel those of two others."""
    n = 64 * 6
    # (first dipole, second, size): tiles (0,2) (0,4) (1,3) and (0,1) (0,3) of the upper triangle
    pairs = [(0, 128, BIG), (1, 256, MIDDLE), (65, 193, TINY), (2, 66, -BIG), (3, 192, -MIDDLE)]

    def run(which):
        pos, mom = _grid(n), np.zeros((n, 3))
        for k, (i, j, size) in enumerate(pairs):
            if k not in which:
                continue
            pos[i] = np.array([8.0 + 12.0 * k, 40.0, 58.0])
            pos[j] = pos[i] + np.array([0.25, -0.125, 0.375])
            mom[i] = (0.375, 0.75, -0.625)
            mom[j] = size * np.array([0.5, -0.875, 0.75])
        return _noalloc(pos, mom, 4.0)[2]

    term = [run([k]) for k in range(5)]
    assert np.array_equal(term[3], -term[0]) and np.array_equal(term[4], -term[1])
    assert np.all(term[2] != 0)
    assert np.array_equal(run(range(5)), term[2])


def test_noalloc_keeps_what_is_not_a_number():
    """Two dipoles at one place, or moments whose products leave FP32: no finite
    number comes out for them, and finite ones for the others."""
    n = 130
    for fault in ("one place", "moments"):
        pos, mom = _grid(n), np.tile(np.array([0.3, 0.4, 0.5]), (n, 1))
        if fault == "one place":
            pos[129] = pos[3]
            bad = [3, 129]
        else:
            mom[[3, 129]] = 3e25
            pos[129] = pos[3] + np.array([1.0, 0.0, 0.0])
            bad = [3, 129]
        F, T, UPT = _noalloc(pos, mom, 4.0)
        assert not np.isfinite(F[bad]).any(), (fault, F[bad])
        assert not np.isfinite(UPT[0]), fault
        if fault == "one place":
            assert not np.isfinite(T[bad]).any()
            rest = [i for i in range(n) if i not in bad]
            assert np.isfinite(F[rest]).all() and np.isfinite(T[rest]).all()


@pytest.mark.parametrize("n", [32, 288, 600])
def test_moment_tensor_of_the_self_terms_in_fp64(n):
    """All rods at one place, moments in opposite pairs: the structure factor is
    zero and the pressure tensor's xy term is the moment tensor's, whose terms
    cancel within a chunk of 256 rods (n = 32), or between two and three."""
    third = {32: 16, 288: 256, 600: 512}[n]  # where the opposite terms stand

    def run(sizes):
        m = np.zeros((n, 3))
        for k, v in enumerate(sizes):
            # products of the same sign in a pair, +-(v, 1) or +-(v, -1)
            at = 4 * k if k < 3 else third + 1 + 4 * (k - 3)
            m[at] = (abs(v), np.sign(v), 0.0)
            m[at + 2] = -m[at]
        dip = np.zeros((n, 1, 5))
        dip[:, 0, 1:4] = m
        dip[:, 0, 4] = 1.0
        st = S.SystemState(np.zeros((n, 3)), np.zeros((n, 3)), np.stack([np.eye(3)] * n), np.zeros((n, 3)),
                           np.full(n, 2.0), np.ones(n), np.ones(n), dip)
        spec = S.SystemSpec(n=n, box=np.full(3, 16.0), alpha=0.4, K_max=2, ksq_max=1)
        with L.Batch([spec], [st]) as bt:
            bt.zero_forces()
            return bt.force_dipK()[1][0]

    alone = run([0.0, 0.0, TINY])
    assert alone[0][1] != 0 and alone[0][1] == alone[1][0]
    got = run([BIG, MIDDLE, TINY, -BIG, -MIDDLE])
    assert got[0][1] == alone[0][1] and got[1][0] == alone[1][0]


def test_field_energy_of_a_moment_across_the_field():
    """mu o . B of moments nearly across the field, where the components' products
    cancel to 2^-44: within five FP64 roundings of the products."""
    rng = np.random.default_rng(11)
    for n in (1, 1, 1, 1, 1, 1, 1, 1, 33):
        x, y = rng.uniform(0.3, 0.9, 2)
        m = np.array([x, y, 0.0])
        B = np.array([y, -x * (1.0 + 2.0 ** -44), 0.0])
        dip = np.zeros((n, 1, 5))
        dip[:, 0, 1:4] = m
        dip[:, 0, 4] = 1.0
        st = S.SystemState(np.arange(3.0 * n).reshape(n, 3) % 29.0, np.zeros((n, 3)), np.stack([np.eye(3)] * n),
                           np.zeros((n, 3)), np.full(n, 2.0), np.ones(n), np.ones(n), dip)
        spec = S.SystemSpec(n=n, box=np.full(3, 30.0), alpha=0.2, K_max=2, ksq_max=1, B=B)
        with L.Batch([spec], [st]) as bt:
            bt.zero_forces()
            U = bt.ext_field()[0]
        exact = -n * float(Fraction(m[0]) * Fraction(B[0]) + Fraction(m[1]) * Fraction(B[1]))
        assert exact != 0.0
        assert abs(U - exact) <= n * 5 * 2.0 ** -53 * (abs(m[0] * B[0]) + abs(m[1] * B[1])), (n, U, exact)
