"""Contexts that are larger than their systems, or used for one system after another:
every build starts from what the trees before it left behind.  Trees against the
oracle (bit-exact) after larger and smaller systems, batches and failed builds; and
a small system's step costs in a large context what it costs in one of its size.
Also the boxes of systems of one block and of several in one batch.
"""
import numpy as np
import pytest

from nns_gb300 import ic
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _joined(systems):
    off = np.concatenate([[0], np.cumsum([len(q.x) for q in systems])])
    b = ic.Bodies(*(np.concatenate([getattr(q, f) for q in systems]) for f in ("x", "y", "z", "vx", "vy", "vz", "m")))
    return b, off


def _build(ctx, systems):
    from nns_gb300.barnes_hut import State
    b, off = _joined(systems)
    ctx.set_systems(off)
    s = State.from_bodies(b)
    ctx.build(s)
    return s


def _check(ctx, systems):
    for j, q in enumerate(systems):
        gt, ot = ctx.export_tree(j), O.build(q.x, q.y, q.z, q.m)
        assert gt["ncells"] == ot.ncells
        for k in ("perm", "root_child", "cell_child", "cell_start", "cell_count", "cell_level", "cell_x", "cell_y",
                  "cell_z", "cell_m"):
            assert np.array_equal(gt[k], getattr(ot, k)), (j, k)


def _failing(n):
    b = ic.plummer(n, seed=n)
    x, y, z = b.x.copy(), b.y.copy(), b.z.copy()
    x[7], y[7], z[7] = x[8], y[8], z[8]  # the same place: NBX_ERR_DEPTH
    return ic.Bodies(x, y, z, b.vx, b.vy, b.vz, b.m)


def test_one_system_after_another(cuda):
    from nns_gb300._lib import NbxError
    from nns_gb300.barnes_hut import Context
    ctx = Context(max_bodies=70000, max_systems=40)
    runs = [[65536], [1000], [3], [70000], [20000], [1, 300, 5000, 2, 257], [66000], [100] * 40, [4097], [1]]
    for j, sizes in enumerate(runs):
        systems = [ic.plummer(k, seed=100 * j + i) for i, k in enumerate(sizes)]
        _build(ctx, systems)
        ctx.sync()
        _check(ctx, systems)
        if j % 3 == 0:
            _build(ctx, [_failing(30000)])
            with pytest.raises(NbxError) as e:
                ctx.sync()
            assert e.value.code == 3  # NBX_ERR_DEPTH


def test_after_a_tree_that_did_not_fit(cuda):
    from nns_gb300._lib import NbxError
    from nns_gb300.barnes_hut import Context
    ctx = Context(max_bodies=5000, node_capacity=5001)
    small = [ic.plummer(2000, seed=5)]
    for _ in range(2):
        _build(ctx, small)
        ctx.sync()
        _check(ctx, small)
        _build(ctx, [ic.plummer(5000, seed=6)])
        with pytest.raises(NbxError) as e:
            ctx.sync()
        assert e.value.code == 4  # NBX_ERR_CAPACITY


def _best_us(fn, reps=30):
    import torch
    best = 1e30
    for _ in range(reps):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        fn()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3)
    return best


@pytest.mark.parametrize("before", [0, 1 << 22])
def test_a_small_system_in_a_large_context(cuda, before):
    """A step of 1000 bodies in a context of 2^24, also after a large system, within
    half as much again of one in a context of 1000 (clearing the whole node pool
    took eight times as long)."""
    from nns_gb300.barnes_hut import Context, State
    b = ic.star_disk(1000)
    us = []
    for cap in (1000, 1 << 24):
        ctx = Context(max_bodies=cap, theta=0.5, eps=0.01, dt=1e-6)
        if before and cap > before:
            _build(ctx, [ic.plummer(before, seed=1)])
            ctx.sync()
        ctx.set_systems([0, 1000])
        s = State.from_bodies(b)
        us.append(_best_us(lambda: ctx.step(s, 1)))
        ctx.sync()
    assert us[1] < 1.5 * us[0], us


def test_boxes_of_a_batch(cuda):
    """Systems of one box block and of many, off centre (the boxes contain the
    origin), with signed zeros: the keys of every system are those of its own box,
    in every build."""
    from nns_gb300.barnes_hut import Context
    systems = []
    for j, k in enumerate([1, 2, 255, 256, 257, 40000, 3, 511, 513, 100000, 1, 8, 20000]):
        b = ic.plummer(k, seed=50 + j)
        sh = [np.float32(3.0 * ((j + a) % 3 - 1)) for a in range(3)]
        x, y, z = b.x + sh[0], b.y + sh[1], b.z + sh[2]
        if j % 2:
            x[0], y[0], z[0] = np.float32(-0.0), np.float32(0.0), np.float32(-0.0)
        systems.append(ic.Bodies(x, y, z, b.vx, b.vy, b.vz, b.m))
    _, off = _joined(systems)
    ctx = Context(max_bodies=int(off[-1]), max_systems=len(systems))
    s = _build(ctx, systems)
    for _ in range(2):
        ctx.build(s)
        ctx.sync()
        keys, perm = ctx.export_keys()
        for j, q in enumerate(systems):
            hi, lo = O.keys(q.x, q.y, q.z, O.bbox(q.x, q.y, q.z), 42)
            o = np.lexsort((lo, hi))
            assert np.array_equal(perm[off[j]:off[j + 1]] - off[j], o), j
            assert np.array_equal(keys[off[j]:off[j + 1]], hi[o]), j


def test_one_kind_of_sort_after_another(cuda):
    """A context holds the lists of its present sort and walks only: systems set one
    after another for every kind (one block's keys, merges, one-sweep and scanned
    radix passes, both walks) sort and walk as in a context of their own."""
    from nns_gb300.barnes_hut import Context
    runs = [[524289], [200], [1000, 40000], [1, 300, 524289, 5000], [30] * 64 + [20000], [1600000], [16384] * 3,
            [600000, 900000, 100], [16385], [3, 5]]
    whole = ic.plummer(1600000, seed=23)
    one = Context(max_bodies=1600000, max_systems=65, theta=1.0, eps=0.1)
    for sizes in runs:
        off = np.concatenate([[0], np.cumsum(sizes)])
        systems = [ic.Bodies(*(np.ascontiguousarray(getattr(whole, f)[a:e])
                               for f in ("x", "y", "z", "vx", "vy", "vz", "m"))) for a, e in zip(off[:-1], off[1:])]
        own = Context(max_bodies=int(off[-1]), max_systems=len(sizes), theta=1.0, eps=0.1)
        got = []
        for ctx in (one, own):
            s = _build(ctx, systems)
            ctx.forces(s)
            ctx.sync()
            got.append(ctx.export_keys() + (s.acc(),))
        for u, v in zip(*got):
            assert np.array_equal(u, v), sizes
