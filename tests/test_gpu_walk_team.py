"""The walk by teams of warps (systems of up to 16384 bodies) beside the walk by
single warps: a batch of both kinds gives every system the bits of its single
run in every mode, group ranges of it sum to the full walk, and the lists and
forces of small and odd systems match the oracle.
"""
import numpy as np
import pytest

from nns_gb300 import ic
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MED_TOL, MAX_TOL = 1e-5, 1e-4  # the walk tests' bounds: rsqrt and summation order differ


def _run(b, off, **kw):
    from nns_gb300.barnes_hut import Context, State
    ctx = Context(max_bodies=int(off[-1]), max_systems=len(off) - 1, theta=0.5, eps=0.01, **kw)
    ctx.set_systems(off)
    s = State.from_bodies(b)
    ctx.build(s)
    ctx.forces(s)
    ctx.sync()
    return ctx, s


@pytest.mark.parametrize("kw", [{}, {"compensated": 1}, {"compensated": 2}, {"multipole": 1},
                                {"multipole": 1, "compensated": 1}, {"leaf_size": 4}],
                         ids=["plain", "split", "kahan", "quad", "quad-split", "buckets"])
def test_batch_of_both_kinds(cuda, kw):
    sizes = [333, 16385, 1, 16384, 4097]
    systems = [ic.plummer(k, seed=21 + j) for j, k in enumerate(sizes)]
    off = np.concatenate([[0], np.cumsum(sizes)])
    b = ic.Bodies(*(np.concatenate([getattr(q, f) for q in systems]) for f in ("x", "y", "z", "vx", "vy", "vz", "m")))
    ctx, s = _run(b, off, **kw)
    acc = s.acc()
    nl, no = ctx.walk_stats()
    for j, q in enumerate(systems):
        c1, s1 = _run(q, np.array([0, sizes[j]]), **kw)
        assert np.array_equal(acc[off[j]:off[j + 1]], s1.acc()), j
        l1, o1 = c1.walk_stats()
        assert np.array_equal(nl[off[j]:off[j + 1]], l1) and np.array_equal(no[off[j]:off[j + 1]], o1), j
    ng = ctx.group_count()
    total = np.zeros_like(acc)
    for a, e in ((0, 7), (7, 400), (400, 400), (400, 830), (830, ng)):
        for t in (s.ax, s.ay, s.az):
            t.zero_()
        ctx.forces_groups(s, a, e - a)
        ctx.sync()
        total += s.acc()
    assert np.array_equal(total, acc)


@pytest.mark.parametrize("n", [1, 2, 9, 31, 33, 97, 1000, 5003])
@pytest.mark.parametrize("stack_depth", [360, 512])
def test_lists_and_forces_match_oracle(cuda, n, stack_depth):
    b = ic.star_disk(n)
    ctx, s = _run(b, np.array([0, n]), stack_depth=stack_depth)
    ot = O.build(b.x, b.y, b.z, b.m)
    theta_ref, eps2 = ctx.constants()
    f = O.forces(b.x, b.y, b.z, b.m, ot, theta_ref, eps2)
    nl, no = ctx.walk_stats()
    assert np.array_equal(nl, f.nlist) and np.array_equal(no, f.nopen)
    a = np.asarray(s.acc(), np.float64)
    rel = np.linalg.norm(a - f.a, axis=1) / np.maximum(np.linalg.norm(f.a, axis=1), 1e-30)
    assert np.median(rel) <= MED_TOL and rel.max() <= MAX_TOL
