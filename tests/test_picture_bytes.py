"""Pixels in which the two halves of a dipole's segment meet: which of them a pixel
shows hangs on the last bits of the segment's ends, which are those of the
expressions in FP32 with one rounding each (centre + length * direction)."""
import numpy as np
import pytest

from mdspherocyl_gb300 import lib as L
from mdspherocyl_gb300 import systems as S

pytestmark = pytest.mark.gpu

TAIL, HEAD = (0, 0, 255), (255, 0, 0)
# seed, rods, packing fraction; view; pixel and its colour
CASES = [
    (462671, 20, 0.2, dict(width=246, height=82, theta=1.235, phi=5.939, dist=20.59, box=False), (128, 34), TAIL),
    (567995, 256, 0.064, dict(width=226, height=53, theta=0.351, phi=2.067, dist=18.9, box=False), (36, 28), TAIL),
    (652289, 513, 0.109, dict(width=258, height=78, theta=1.158, phi=1.982, dist=16.9, box=True), (21, 18), TAIL),
    (123948, 256, 0.123, dict(width=91, height=103, theta=0.76, phi=4.392, dist=26.56, box=True), (62, 21), TAIL),
    (75083, 256, 0.117, dict(width=163, height=40, theta=2.709, phi=4.569, dist=9.79, box=True), (98, 31), HEAD),
    (166044, 513, 0.126, dict(width=235, height=56, theta=1.826, phi=5.803, dist=23.99, box=True), (132, 6), TAIL),
]


@pytest.mark.parametrize("k", range(len(CASES)))
def test_pixels_between_the_halves_of_a_dipole(k):
    seed, n, phi, view, (x, y), colour = CASES[k]
    st, box = S.make_system(n=n, phi=phi, lengths=np.full(n, 3.0), mu=np.full(n, 1.2), seed=seed)
    st.dip = np.zeros((n, 2, 5))
    for w in range(2):
        st.dip[:, w] = (0.5 * w - 0.7, 0.6, 0.0, 0.8, 0.5 + 0.2 * w)
    spec = S.SystemSpec(n=n, box=box, alpha=6.0 / float(box[0]), K_max=2, ksq_max=1)
    with L.Batch([spec], [st]) as bt:
        img = np.asarray(bt.render(0, **view))
    assert tuple(int(c) for c in img[y, x]) == colour
