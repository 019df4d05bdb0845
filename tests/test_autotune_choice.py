"""What a tuning run chooses: the fastest mapping of those it timed, and for the
WCA evaluation's grid the smallest that no larger one beats by 5% (a grid holds
registers from the step's other chains, which a kernel timed alone does not
show)."""
import re

import numpy as np
import pytest

from mdspherocyl_gb300 import lib as L
from mdspherocyl_gb300 import systems as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,copies", [(256, 1), (32768, 1), (700, 24), (128, 330)])
def test_the_choice_is_the_fastest(n, copies):
    st, box = S.make_system(n=n, phi=0.1, lengths=np.full(n, 3.0), mu=np.full(n, 1.2), seed=17)
    spec = S.SystemSpec(n=n, box=box, alpha=6.0 / float(box[0]), K_max=6, ksq_max=27)
    with L.Batch([spec] * copies, [st] * copies) as bt:
        for _ in range(5):
            t = bt.autotune(force=True)
            times = {}
            for what, v, ms in re.findall(r"(\w+)=(\d+) ([\d.]+) ms;", t["log"]):
                times.setdefault(what, []).append((int(v), float(ms)))
            for what in ("rp_warps", "rsum_threads", "kg_scalar"):
                chosen = dict(times[what])[t[what]]
                assert chosen <= min(ms for _, ms in times[what]) + 1.01e-4, (what, times[what], t[what])
            wca = times["wca_blocks"]
            assert 0.95 * dict(wca)[t["wca_blocks"]] <= min(ms for _, ms in wca) + 1.01e-4, (wca, t["wca_blocks"])
