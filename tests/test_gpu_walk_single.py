"""The walk by single warps (k_walk2), which systems above the teams' size take: every
buffer variant, accumulation mode, launch shape and option against the oracle.
"""
import numpy as np
import pytest

from nns_gb300 import ic
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MED_TOL, MAX_TOL = 1e-5, 1e-4  # the walk tests' bounds: rsqrt and summation order differ


@pytest.mark.parametrize("variant,slots", [(0, 64), (1, 128), (3, 96)])
def test_uncompensated_stretch_of_the_split_mode(cuda, variant, slots):
    """compensated = 1 sums plainly within a round and compensates across rounds: a
    round never holds more candidates than its buffers did when the mode was made."""
    from nns_gb300.barnes_hut import Context, State
    b = ic.plummer(40000)
    ctx = Context(max_bodies=len(b.x), theta=0.5, eps=0.01, compensated=1)
    ctx.set_walk(8, variant)
    ctx.set_systems([0, len(b.x)])
    s = State.from_bodies(b)
    ctx.build(s)
    ctx.forces(s)
    ctx.sync()
    info = ctx.tree_info()
    assert info["candidates"] <= slots * info["rounds"]


@pytest.mark.parametrize("n", [255, 256, 257, 258, 16383, 16384, 16385])
def test_batches_where_the_walks_change(cuda, n):
    """Systems of up to 256 bodies and of more than 2^14 are walked by single warps,
    those between by teams: a batch with sizes on both sides gives every system the
    bits of its single run and the oracle's lists."""
    from nns_gb300.barnes_hut import Context, State
    sizes = [n, 100, 1000, n, 1, 20000]
    systems = [ic.plummer(k, seed=70 + j) for j, k in enumerate(sizes)]
    off = np.concatenate([[0], np.cumsum(sizes)])

    def run(parts, o):
        b = ic.Bodies(*(np.concatenate([getattr(q, f) for q in parts]) for f in ("x", "y", "z", "vx", "vy", "vz", "m")))
        ctx = Context(max_bodies=int(o[-1]), max_systems=len(parts), theta=0.5, eps=0.01)
        ctx.set_systems(o)
        s = State.from_bodies(b)
        for _ in range(3):  # (the group counter of the single-warp walk is left as found)
            ctx.build(s)
            ctx.forces(s)
            ctx.forces(s)
        ctx.sync()
        return ctx, s

    ctx, s = run(systems, off)
    nl, no = ctx.walk_stats()
    for j, q in enumerate(systems):
        c1, s1 = run([q], np.array([0, sizes[j]]))
        assert np.array_equal(s.acc()[off[j]:off[j + 1]], s1.acc()), j
        t, e2 = c1.constants()
        f = O.forces(q.x, q.y, q.z, q.m, O.build(q.x, q.y, q.z, q.m), t, e2)
        assert np.array_equal(nl[off[j]:off[j + 1]], f.nlist) and np.array_equal(no[off[j]:off[j + 1]], f.nopen), j
        rel = np.linalg.norm(s1.acc() - f.a, axis=1) / np.maximum(np.linalg.norm(f.a, axis=1), 1e-30)
        if sizes[j] > 1:
            assert np.median(rel) <= MED_TOL and rel.max() <= MAX_TOL, j
