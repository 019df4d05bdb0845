"""When a step builds the Verlet list: by how far the rods have moved since the
last build, whatever was asked of the batch in between."""
import ctypes

import numpy as np
import pytest

from mdspherocyl_gb300 import lib as L
from mdspherocyl_gb300 import systems as S

pytestmark = pytest.mark.gpu


def _system(n, seed):
    st, box = S.make_system(n=n, phi=0.08, lengths=np.full(n, 3.0), mu=np.full(n, 1.2), seed=seed)
    return S.SystemSpec(n=n, box=box, alpha=6.0 / float(box[0]), K_max=4, ksq_max=9), st


CALLS = {
    "neigh_list": lambda bt: bt.neigh_list(),
    "check_list": lambda bt: bt.check_list(),
    "correlations": lambda bt: bt.correlations(0.2),
    "order_params": lambda bt: bt.order_params(),
    "renorm": lambda bt: bt.renorm(),
}


@pytest.mark.parametrize("call", list(CALLS))
def test_a_configuration_looked_at_is_not_a_configuration_stepped(call):
    """A state uploaded far away, looked at, and (but for neigh_list, whose list is
    that state's) the old one uploaded again: the next step has a list that stands
    and builds none."""
    spec, st = _system(300, 5)
    with L.Batch([spec], [st]) as bt:
        builds = bt.step(3)[0]["list_builds"]
        d = bt.download(0)
        arrays = [np.ascontiguousarray(d[k]) for k in ("r", "p", "O", "l", "F", "T")]
        away = [arrays[0] + np.array([4.0, 0.0, 0.0])] + arrays[1:]
        bt.upload_all(*away)
        CALLS[call](bt)
        if call != "neigh_list":
            bt.upload_all(*arrays)
        obs = bt.step(1)[0]
        assert obs["list_builds"] == builds
        # and the step after a real move does build one
        d = bt.download(0)
        bt.upload_all(*[np.ascontiguousarray(d[k]) + (np.array([0.0, 4.0, 0.0]) if k == "r" else 0.0)
                        for k in ("r", "p", "O", "l", "F", "T")])
        assert bt.step(1)[0]["list_builds"] == builds + 1


def test_a_system_left_out_of_a_force_evaluation():
    """Forces evaluated for one system only: the other's state of that moment does
    not count for its next step."""
    systems = [_system(200, 6), _system(260, 7)]
    with L.Batch([s for s, _ in systems], [t for _, t in systems]) as bt:
        builds = bt.step(3)[0]["list_builds"]
        d = [bt.download(k) for k in range(2)]

        def up(k, shift, forces):
            arrays = [d[k]["r"] + shift] + [d[k][f] for f in ("p", "O", "l") + (("F", "T") if forces else ())]
            hs = bt._hoststate(*arrays)
            bt._check(bt.lib.mdsc_upload(bt.h, k, ctypes.byref(hs)), "mdsc_upload")

        up(0, np.array([4.0, 0.0, 0.0]), True)
        up(1, 0.0, False)
        bt.observe()
        up(0, 0.0, True)
        assert bt.step(1)[0]["list_builds"] == builds
