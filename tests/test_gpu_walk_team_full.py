"""Batches that fill the GPU: the walk by teams is done by one warp per group there,
which takes the four warps' shares in turn.  Every system keeps the bits of its
single run, in every mode, and the oracle's lists.
"""
import numpy as np
import pytest

from nns_gb300 import ic
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _run(systems, off, pot=False, **kw):
    from nns_gb300.barnes_hut import Context, State
    b = ic.Bodies(*(np.concatenate([getattr(q, f) for q in systems]) for f in ("x", "y", "z", "vx", "vy", "vz", "m")))
    ctx = Context(max_bodies=int(off[-1]), max_systems=len(systems), theta=kw.pop("theta", 0.5), eps=0.01, **kw)
    ctx.set_systems(off)
    s = State.from_bodies(b)
    ctx.build(s)
    phi = ctx.potential(s) if pot else None
    ctx.forces(s)
    ctx.sync()
    return ctx, s, phi


# mean sizes on both sides of the rule's ends: 300 (12 groups per SM), 1300, 6000 bodies
SIZES = {"small": [257, 300, 331] * 120, "mid": [1000, 1200, 1500, 1411] * 25, "large": [5003, 7000, 6001] * 45}


@pytest.mark.parametrize("name", list(SIZES))
@pytest.mark.parametrize("kw", [{}, {"compensated": 1}, {"compensated": 2}, {"multipole": 1},
                                {"multipole": 1, "compensated": 1}, {"multipole": 1, "compensated": 2}, {"leaf_size": 4},
                                {"theta": 0.15}, {"theta": 0.15, "stack_depth": 360}],
                         ids=["plain", "split", "kahan", "quad", "quad-split", "quad-kahan", "buckets", "opened",
                              "full-stack"])
def test_full_batches_equal_single_runs(cuda, name, kw):
    sizes = SIZES[name]
    kinds = sorted(set(sizes))
    one = {k: (ic.plummer if k % 2 else ic.star_disk)(k, seed=k) for k in kinds}
    off = np.concatenate([[0], np.cumsum(sizes)])
    ctx, s, phi = _run([one[k] for k in sizes], off, pot=True, **kw)
    acc = s.acc()
    nl, no = ctx.walk_stats()
    for k in kinds:
        c1, s1, phi1 = _run([one[k]], np.array([0, k]), pot=True, **kw)
        l1, o1 = c1.walk_stats()
        for j in [j for j, v in enumerate(sizes) if v == k]:
            a, e = off[j], off[j + 1]
            assert np.array_equal(acc[a:e], s1.acc()) and np.array_equal(phi[a:e], phi1), (k, j)
            assert np.array_equal(nl[a:e], l1) and np.array_equal(no[a:e], o1), (k, j)


def test_lists_match_oracle(cuda):
    sizes = [333] * 400
    systems = [ic.plummer(k, seed=j) for j, k in enumerate(sizes)]
    off = np.concatenate([[0], np.cumsum(sizes)])
    ctx, s, _ = _run(systems, off)
    nl, no = ctx.walk_stats()
    t, e2 = ctx.constants()
    for j in range(0, 400, 37):
        q = systems[j]
        f = O.forces(q.x, q.y, q.z, q.m, O.build(q.x, q.y, q.z, q.m), t, e2)
        a, e = off[j], off[j + 1]
        assert np.array_equal(nl[a:e], f.nlist) and np.array_equal(no[a:e], f.nopen)
        rel = np.linalg.norm(s.acc()[a:e] - f.a, axis=1) / np.linalg.norm(f.a, axis=1)
        assert np.median(rel) <= 1e-5 and rel.max() <= 1e-4
