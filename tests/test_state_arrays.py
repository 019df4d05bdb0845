"""State arrays on their way between host and device: arrays that an upload still
reads are left alone by a download, arrays that are missing are refused, and the
call that zeroes the forces has done so when it returns."""
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


@pytest.mark.parametrize("missing", range(4), ids=["r", "p", "O", "l"])
@pytest.mark.parametrize("n", [64, 9000])
def test_missing_arrays_are_refused(n, missing):
    """r, p, O and l are needed, in the upload of a state and in a step with one;
    the batch's state and forces stay as they were."""
    st, box = S.make_system(n=n, phi=0.05, lengths=np.full(n, 3.0), mu=np.full(n, 1.2), seed=8)
    spec = S.SystemSpec(n=n, box=box, alpha=6.0 / float(box[0]), K_max=2, ksq_max=1)
    arrays = [np.ascontiguousarray(np.asarray(a, dtype=np.float64)) + 0.5 for a in (st.r, st.p, st.O, st.l)]
    arrays += [np.full((n, 3), 9.0), np.full((n, 3), 9.0)]
    arrays[missing] = None
    with L.Batch([spec], [st]) as bt:
        bt.step(1)
        before = bt.download(0)
        with pytest.raises(L.MdscError):
            bt.upload_all(*arrays)
        with pytest.raises(L.MdscError):
            bt.step_io(dict(zip("rpOlFT", arrays)), 1, None)
        after = bt.download(0)
    for k in ("r", "p", "O", "l", "F", "T"):
        assert np.array_equal(before[k], after[k]), k


def test_zero_forces_waits():
    """The call returns with the forces zero, as the other function-level calls
    return with their results."""
    import torch

    spec, st, host = _big()
    with L.Batch([spec], [st]) as bt:
        bt.upload_all(*host)
        stream = torch.cuda.ExternalStream(bt.lib.mdsc_stream(bt.h))
        _backlog(bt, host)
        assert not stream.query()
        bt.zero_forces()
        assert stream.query()
        d = bt.download(0)
    assert not d["F"].any() and not d["T"].any()
