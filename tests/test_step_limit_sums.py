"""The observables of a system that has reached its step limit are those of its
last step, every sum of them, in batches small and large (the per-system sums
run in several blocks each, the last of them when others have long finished)."""
import numpy as np
import pytest

from mdspherocyl_gb300 import lib as L
from mdspherocyl_gb300 import systems as S

pytestmark = pytest.mark.gpu

KEYS = ("U_ss", "W_ss", "U_dipR", "U_dipK", "U_ext", "K", "PT_ss", "PT_dipR", "PT_dipK", "PT_kin", "xi", "G1", "G2", "M",
        "step")


def _system(n, seed):
    st, box = S.make_system(n=n, phi=0.1, lengths=np.full(n, 3.0), mu=np.full(n, 1.2), seed=seed)
    return S.SystemSpec(n=n, box=box, alpha=6.0 / float(box[0]), K_max=4, ksq_max=9, B=np.array([0.2, 0.0, -0.1])), st


@pytest.mark.parametrize("copies", [1, 40, 700])
@pytest.mark.parametrize("calls", [(5,), (2, 3), (1, 1, 1, 1, 1)])
def test_observables_at_the_limit(copies, calls):
    """Three systems of different sizes, `copies` times over, with limits 1, 2 and 4
    (one of them inside a pair of steps) in a run of five."""
    systems = [_system(n, 30 + n) for n in (20, 90, 40)]
    limits = (1, 2, 4)
    want = []
    for (spec, st), lim in zip(systems, limits):
        with L.Batch([spec], [st]) as bt:
            for _ in range(lim):
                o = bt.step(1)[0]
            want.append(o)
    with L.Batch([s for s, _ in systems] * copies, [t for _, t in systems] * copies) as bt:
        for k in range(3 * copies):
            bt.set_step_limit(k, limits[k % 3])
        for n in calls:
            obs = bt.step(n)
    for k in range(3 * copies):
        for key in KEYS:
            assert np.array_equal(np.asarray(obs[k][key]), np.asarray(want[k % 3][key])), (k, key)
