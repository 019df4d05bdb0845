"""State arrays on their way between host and device: arrays that an upload still
reads are left alone by a download."""
import numpy as np
import pytest

from mdspherocyl_gb300 import lib as L
from mdspherocyl_gb300 import systems as S

pytestmark = pytest.mark.gpu

WIDTH = (3, 3, 9, 3, 3, 3)  # r, p, O, l, F, T
N = 32768


def _big():
    """The 32,768-rod system and its state arrays in pinned memory."""
    import torch

    spec, st = S.plain_c2()
    assert st.n == N
    host = [torch.empty(N, w, dtype=torch.float64, pin_memory=True).numpy() for w in WIDTH]
    rng = np.random.default_rng(3)
    for x, y in zip(host, (st.r, st.p, st.O, st.l)):
        x[...] = np.asarray(y).reshape(N, -1)
    for x in host[4:]:
        x[...] = rng.normal(size=x.shape)
    return spec, st, host


def _backlog(bt, host):
    """Uploads that keep the batch's stream busy for a millisecond: 6.3 MB each."""
    for _ in range(60):
        bt.upload_all(*host)


@pytest.mark.parametrize("plain", [0, 2])
def test_a_download_leaves_arrays_that_an_upload_reads(plain):
    """An upload from pinned arrays returns at once; the download into the same
    arrays (but one, which is plain memory) finds in them what went up."""
    import torch

    spec, st, other = _big()
    host = [torch.from_numpy(x + 1.0).pin_memory().numpy() for x in other]
    want = [x.copy() for x in host]
    with L.Batch([spec], [st]) as bt:
        _backlog(bt, other)
        bt.upload_all(*host)
        into = list(host)
        into[plain] = np.full_like(host[plain], 5.0)
        bt.download_all(*into)
        for got, x in zip(into, want):
            assert np.array_equal(got, x)


def test_a_download_into_the_plain_arrays_just_uploaded():
    spec, st, other = _big()
    host = [x + 1.0 for x in other]
    want = [x.copy() for x in host]
    with L.Batch([spec], [st]) as bt:
        _backlog(bt, other)
        bt.upload_all(*host)
        bt.download_all(*host)
        for got, x in zip(host, want):
            assert np.array_equal(got, x)
