"""The WCA pairs' evaluation for large batches (a thread per pair, above 1200 rows
of 32 rods) in every branch of the segment distance: the hand-built
configurations, as often as it takes, against the oracle and against the form
that small batches take."""
import numpy as np
import pytest

import hand_configs as H
import oracle
from mdspherocyl_gb300 import lib as L
from mdspherocyl_gb300 import systems as S

pytestmark = pytest.mark.gpu

COPIES = 100  # 1300 systems of a row each


def test_hand_configs_in_a_large_batch(orc):
    confs = H.build()
    assert COPIES * len(confs) > 1200
    states, specs = [], []
    for c in confs:
        n = len(c["length"])
        states.append(S.SystemState(c["r"], np.zeros((n, 3)), c["O"], np.zeros((n, 3)), c["length"], c["dia"],
                                    np.ones(n), np.zeros((n, 1, 5))))
        specs.append(S.SystemSpec(n=n, box=c["box"], alpha=6.0 / H.BOX, K_max=2, ksq_max=1, min_s=0.6))

    def run(copies):
        with L.Batch(specs * copies, states * copies) as bt:
            bt.zero_forces()
            U, W, PT = bt.force_sc()
            which = list(range(len(confs))) + list(range(len(U) - len(confs), len(U)))
            return [(U[k], W[k], PT[k].copy(), bt.download(k)) for k in which]

    small, large = run(1), run(COPIES)
    for k, (u, w, pt, d) in enumerate(large):
        c = confs[k % len(confs)]
        n = len(c["length"])
        s = oracle.System(c["r"], np.zeros((n, 3)), c["O"], np.zeros((n, 3)), c["length"], c["dia"], np.ones(n),
                          np.zeros((n, 1, 5)), c["box"])
        ok, uo, wo, pto = orc.force_sc(s, 3.0, 3.5)
        scale = max(1.0, np.abs(s.F).max(), np.abs(s.T).max())
        assert abs(u - uo) <= 1e-12 * max(1.0, abs(uo)), (c["members"], u, uo)
        assert abs(w - wo) <= 1e-12 * max(1.0, abs(wo)), (c["members"], w, wo)
        assert np.abs(pt - pto).max() <= 1e-12 * max(1.0, np.abs(pto).max()), c["members"]
        assert np.abs(d["F"] - s.F).max() <= 1e-12 * scale, (c["members"], d["F"], s.F)
        assert np.abs(d["T"] - s.T).max() <= 1e-12 * scale, (c["members"], d["T"], s.T)
        assert np.array_equal(d["F"], small[k % len(confs)][3]["F"]), c["members"]
        assert np.array_equal(d["T"], small[k % len(confs)][3]["T"]), c["members"]
