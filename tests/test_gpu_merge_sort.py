"""The merging sort of small and mid-size systems against NumPy's stable sort of the
42-level keys, at the edges of its runs (1024 keys, sorted in quarters of 256), of
its merging launches (16 runs each) and past them (radix); orders of input that
leave the expected stretches (sorted, reversed, blockwise) and keys with long
equal runs included.  Batches mix systems of every kind.
"""
import numpy as np
import pytest

from nns_gb300 import ic
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _arrange(b, how, rng):
    n = len(b.x)
    hi, lo = _keys(b)
    o = np.lexsort((lo, hi))
    if how == "reversed":
        o = o[::-1]
    elif how == "blocks":  # sorted blocks of 4096 in a shuffled order
        k = [o[i:i + 4096] for i in range(0, n, 4096)]
        o = np.concatenate([k[i] for i in rng.permutation(len(k))])
    elif how == "shuffled":
        o = rng.permutation(n)
    return ic.Bodies(*(np.ascontiguousarray(a[o]) for a in (b.x, b.y, b.z, b.vx, b.vy, b.vz, b.m)))


def _keys(b):
    bb = O.bbox(b.x, b.y, b.z)
    return O.keys(b.x, b.y, b.z, bb, 42)


def _check(ctx, off, systems):
    keys, perm = ctx.export_keys()
    for j, b in enumerate(systems):
        hi, lo = _keys(b)
        o = np.lexsort((lo, hi))
        assert np.array_equal(perm[off[j]:off[j + 1]] - off[j], o), j
        assert np.array_equal(keys[off[j]:off[j + 1]], hi[o]), j


@pytest.mark.parametrize("how", ["shuffled", "sorted", "reversed", "blocks"])
@pytest.mark.parametrize("n", [1, 255, 257, 1024, 1025, 4099, 16384, 16385, 131071, 262144, 262145, 1048577])
def test_sort_matches_numpy(cuda, n, how):
    from nns_gb300.barnes_hut import Context, State
    b = _arrange(ic.plummer(n, seed=n), how, np.random.default_rng(n))
    ctx = Context(max_bodies=n)
    ctx.set_systems([0, n])
    ctx.build(State.from_bodies(b))
    ctx.sync()
    _check(ctx, [0, n], [b])


def test_equal_keys_keep_their_order(cuda):
    """A third of the bodies in a knot a few 21-level cells wide: long runs of equal
    63-bit keys, ordered by their deeper levels."""
    from nns_gb300.barnes_hut import Context, State
    n = 30000
    rng = np.random.default_rng(3)
    b = ic.plummer(n, seed=3)
    x = np.array(b.x)
    k = rng.permutation(n)[: n // 3]
    x[k] = np.float32(0.5) + np.arange(len(k), dtype=np.float32) * np.float32(2.0 ** -24)
    b = ic.Bodies(x, b.y, b.z, b.vx, b.vy, b.vz, b.m)
    y, z = np.array(b.y), np.array(b.z)
    y[k] = 0.25
    z[k] = 0.125
    b = ic.Bodies(x, y, z, b.vx, b.vy, b.vz, b.m)
    ok = np.unique(np.stack([x, y, z], 1), axis=0, return_index=True)[1]
    b = ic.Bodies(*(np.ascontiguousarray(a[np.sort(ok)]) for a in (b.x, b.y, b.z, b.vx, b.vy, b.vz, b.m)))
    n = len(b.x)
    hi, _ = _keys(b)
    assert len(np.unique(hi)) < n  # equal 63-bit keys are there
    ctx = Context(max_bodies=n)
    ctx.set_systems([0, n])
    ctx.build(State.from_bodies(b))
    ctx.sync()
    _check(ctx, [0, n], [b])


@pytest.mark.parametrize("sizes", [[1, 300, 16384, 2, 257], [5, 70000, 256, 20000]])
def test_batches(cuda, sizes):
    from nns_gb300.barnes_hut import Context, State
    systems = [ic.plummer(k, seed=11 + j) for j, k in enumerate(sizes)]
    off = np.concatenate([[0], np.cumsum(sizes)])
    b = ic.Bodies(*(np.concatenate([getattr(q, f) for q in systems]) for f in ("x", "y", "z", "vx", "vy", "vz", "m")))
    ctx = Context(max_bodies=int(off[-1]), max_systems=len(sizes))
    ctx.set_systems(off)
    ctx.build(State.from_bodies(b))
    ctx.sync()
    _check(ctx, off, systems)
