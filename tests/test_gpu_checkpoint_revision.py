"""A checkpoint holds the revision of the walk's order of summation, which fixes the
force bits beside the recorded settings: a file of another revision (or from before
there were any) is restored, and says that the run does not continue bit for bit.
"""
import warnings

import numpy as np
import pytest

from nns_gb300 import ic

pytestmark = pytest.mark.gpu


def _fnv1a(data, h=1469598103934665603):
    for v in data:
        h = ((h ^ v) * 1099511628211) & 0xFFFFFFFFFFFFFFFF
    return h


def _with_revision(buf, revision):
    """The checkpoint with another revision (int32 at byte 68; header hash at 72, over
    the bytes before it and the offsets from byte 80)."""
    b = buf.copy()
    b[68:72] = np.frombuffer(np.int32(revision).tobytes(), np.uint8)
    nsys = int(np.frombuffer(b[12:16].tobytes(), np.int32)[0])
    b[72:80] = np.frombuffer(np.uint64(_fnv1a(b[80:80 + 8 * (nsys + 1)].tolist(), _fnv1a(b[:72].tolist()))).tobytes(),
                             np.uint8)
    return b


@pytest.mark.parametrize("revision", [None, 0, 7])
def test_revisions(cuda, revision):
    from nns_gb300.barnes_hut import Context, State
    b = ic.plummer(3000)
    ctx = Context(max_bodies=3000, theta=0.5, eps=0.01)
    ctx.set_systems([0, 3000])
    s = State.from_bodies(b)
    ctx.step(s, 2)
    ctx.sync()
    saved = ctx.checkpoint(s)
    other = Context(max_bodies=3000, theta=0.7, eps=0.02)
    r = State.empty(3000)
    with warnings.catch_warnings(record=True) as w:
        warnings.simplefilter("always")
        other.restore(r, saved if revision is None else _with_revision(saved, revision))
    assert [str(v.message).split(":")[0] for v in w] == ([] if revision is None else ["checkpoint"])
    for u, v in zip(s.host(), r.host()):
        assert np.array_equal(u, v)
    for c, q in ((ctx, s), (other, r)):
        c.step(q, 1)
        c.sync()
    for u, v in zip(s.host(), r.host()):
        assert np.array_equal(u, v)
