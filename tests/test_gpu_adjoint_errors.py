"""Recording lists that overflow (nbx_adjoint_create's list_capacity): the adjoint
of a batch of small systems, whose walk groups outnumber the blocks that the GPU
holds at once, so that blocks of one launch start after others have reported the
full list.  The forward reports NBX_ERR_CAPACITY and nothing else, the context goes on
as a fresh one does, and passes over a tape whose recording was stopped stay
within it.
"""
import numpy as np
import pytest

from nns_gb300 import ic

pytestmark = pytest.mark.gpu

NBX_ERR_CAPACITY = 4


def _batch(sizes):
    parts = [ic.plummer(k, seed=ic.SEED0 + 40 + j) for j, k in enumerate(sizes)]
    off = np.concatenate([[0], np.cumsum(sizes)])
    b = ic.Bodies(*(np.concatenate([getattr(q, f) for q in parts]) for f in ("x", "y", "z", "vx", "vy", "vz", "m")))
    return b, off


def _context(off):
    from nns_gb300.barnes_hut import Context
    ctx = Context(max_bodies=int(off[-1]), max_systems=len(off) - 1, theta=0.5, eps=0.01, dt=1e-3)
    ctx.set_systems(off)
    return ctx


def _stepped(ctx, b):
    from nns_gb300.barnes_hut import State
    s = State.from_bodies(b)
    ctx.step(s, 1)
    ctx.sync()
    return s.host() + (s.acc(),)


@pytest.mark.parametrize("sizes", [[4000] * 24, [20000] * 12], ids=["teams", "single-warps"])
def test_full_lists_are_reported(cuda, sizes):
    import torch
    from nns_gb300._lib import NbxError
    from nns_gb300.adjoint import Adjoint
    from nns_gb300.barnes_hut import State
    b, off = _batch(sizes)  # 3000 and 7500 groups
    ctx = _context(off)
    target = torch.zeros(3, int(off[-1]), device="cuda")
    adj = Adjoint(ctx, 3, 1, 64)
    for _ in range(3):
        with pytest.raises(NbxError) as e:
            adj.forward(State.from_bodies(b), target)
        assert e.value.code == NBX_ERR_CAPACITY
    for got, want in zip(_stepped(ctx, b), _stepped(_context(off), b)):
        assert np.array_equal(got, want)


def test_passes_over_a_stopped_recording(cuda):
    """The first recorded step overflows, so the later steps' trees are built empty
    and their lists never written: the reverse pass and the FP64 replay over that
    tape have nothing to index by but what the adjoint's creation left there."""
    import torch
    from nns_gb300._lib import NbxError
    from nns_gb300.adjoint import Adjoint
    from nns_gb300.barnes_hut import State
    b, off = _batch([4000] * 4)
    n = int(off[-1])
    ctx = _context(off)
    target = torch.zeros(3, n, device="cuda")
    adj = Adjoint(ctx, 4, 4, 64)
    s = State.from_bodies(b)
    with pytest.raises(NbxError) as e:
        adj.forward(s, target)
    assert e.value.code == NBX_ERR_CAPACITY
    g = adj.backward(s)
    torch.cuda.synchronize()
    assert [t.shape[-1] for t in g] == [n] * 3
    with pytest.raises(NbxError) as e:
        adj.record(s)
    assert e.value.code == NBX_ERR_CAPACITY
    adj.replay_fp64(torch.zeros(7, n, dtype=torch.float64, device="cuda"))
    torch.cuda.synchronize()
    for got, want in zip(_stepped(ctx, b), _stepped(_context(off), b)):
        assert np.array_equal(got, want)
