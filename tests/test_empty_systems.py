"""A batch whose systems hold no rods: every call goes through, with zeros."""
import numpy as np
import pytest

from mdspherocyl_gb300 import lib as L
from mdspherocyl_gb300 import systems as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("systems", [1, 3])
def test_only_empty_systems(systems):
    st = S.SystemState(np.zeros((0, 3)), np.zeros((0, 3)), np.zeros((0, 3, 3)), np.zeros((0, 3)), np.zeros(0),
                       np.zeros(0), np.zeros(0), np.zeros((0, 1, 5)))
    spec = S.SystemSpec(n=0, box=np.full(3, 12.0), alpha=0.5, K_max=3, ksq_max=4)
    with L.Batch([spec] * systems, [st] * systems) as bt:
        bt.zero_forces()
        for U in (bt.force_sc()[0], bt.force_dipR()[0], bt.force_dipK()[0], bt.ext_field()):
            assert not np.any(U)
        obs = bt.observe()
        obs = bt.step(5)
        lab, nc = bt.clust_conf(0)
        bt.neigh_list()
        d = bt.download(0)
    assert [o["step"] for o in obs] == [5] * systems
    assert all(o[k] == 0.0 for o in obs for k in ("U_ss", "U_dipR", "U_dipK", "U_ext"))
    assert nc == 0 and len(lab) == 0 and d["r"].shape == (0, 3)
