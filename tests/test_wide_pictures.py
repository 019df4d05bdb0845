"""Low, wide pictures, whose blocks of 16 x 8 pixels span more than a right angle:
a pixel is the middle one of the 15 x 15 that the same view has in a picture 15
times as large, whose blocks span little.  Rods only (the lines' width goes by
the pixel)."""
import numpy as np
import pytest

from mdspherocyl_gb300 import lib as L
from mdspherocyl_gb300 import systems as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height", [(17, 1), (20, 2), (24, 3), (49, 3), (122, 3), (300, 4), (16, 8), (48, 40)])
def test_a_wide_picture_is_the_middle_of_a_large_one(width, height):
    st, box = S.make_system(n=200, phi=0.05, lengths=np.full(200, 3.0), mu=np.full(200, 1.2), seed=12)
    st.r = st.r - 0.5 * box  # around the camera
    spec = S.SystemSpec(n=200, box=box, alpha=6.0 / float(box[0]), K_max=2, ksq_max=1)
    rng = np.random.default_rng(width)
    off = total = 0
    with L.Batch([spec], [st]) as bt:
        for _ in range(100):
            v = dict(theta=float(rng.uniform(0.3, 2.8)), phi=float(rng.uniform(0, 6)), dist=float(rng.uniform(0.3, 3.0)),
                     dipoles=False, box=False)
            small = np.asarray(bt.render(0, width=width, height=height, **v)).astype(int)
            large = np.asarray(bt.render(0, width=15 * width, height=15 * height, **v)).astype(int)[7::15, 7::15]
            off += (np.abs(small - large).max(axis=-1) > 3).sum()
            total += width * height
    # rays an ulp apart on the outline of a rod
    assert off <= 0.001 * total, (off, total)
