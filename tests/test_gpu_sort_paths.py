"""Every way the body keys are sorted, against NumPy's stable sort of the 42-level
keys: batches with many systems of one block's keys (a launch of their own) beside
larger ones; the batches on both sides of the rule that picks merges or radix passes;
and the radix passes of batches, one-sweep and scanned, with both digit widths.
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


def _built(systems, **kw):
    from nns_gb300.barnes_hut import Context, State
    b, off = _joined(systems)
    ctx = Context(max_bodies=int(off[-1]), max_systems=len(systems), **kw)
    ctx.set_systems(off)
    s = State.from_bodies(b)
    ctx.build(s)
    ctx.sync()
    return ctx, s, off


def _check(ctx, off, systems):
    keys, perm = ctx.export_keys()
    for j, b in enumerate(systems):
        hi, lo = O.keys(b.x, b.y, b.z, O.bbox(b.x, b.y, b.z), 42)
        o = np.lexsort((lo, hi))
        assert np.array_equal(perm[off[j]:off[j + 1]] - off[j], o), j
        assert np.array_equal(keys[off[j]:off[j + 1]], hi[o]), j


SMALL = [1, 2, 3, 31, 32, 33, 63, 64, 65, 127, 128, 129, 200, 255, 256, 7] * 5


@pytest.mark.parametrize("more", [[], [257], [1000, 20000], [300] * 40], ids=["alone", "257", "larger", "many"])
def test_many_systems_of_one_block(cuda, more):
    sizes = [k for p in zip(SMALL, more + [0] * len(SMALL)) for k in p if k]
    systems = [ic.plummer(k, seed=300 + j) for j, k in enumerate(sizes)]
    ctx, _, off = _built(systems)
    _check(ctx, off, systems)


def test_equal_keys_in_one_block(cuda):
    """Bodies in a few 21-level cells, in a shuffled order: equal 63-bit keys keep
    their bodies' order until their deeper levels decide."""
    systems = []
    for j in range(70):
        b = ic.plummer(200, seed=j)
        x, y, z = b.x.copy(), b.y.copy(), b.z.copy()
        k = np.random.default_rng(j).permutation(200)[:64]
        x[k] = np.float32(0.5) + np.arange(64, dtype=np.float32) * np.float32(2.0 ** -24)
        y[k], z[k] = 0.25, 0.125
        x[k] = np.unique(x[k])[np.arange(64) % len(np.unique(x[k]))]
        p = np.unique(np.stack([x, y, z], 1), axis=0, return_index=True)[1]
        systems.append(ic.Bodies(*(np.ascontiguousarray(a[np.sort(p)]) for a in (x, y, z, b.vx, b.vy, b.vz, b.m))))
    hi, _ = O.keys(systems[0].x, systems[0].y, systems[0].z, O.bbox(systems[0].x, systems[0].y, systems[0].z), 42)
    assert len(np.unique(hi)) < len(hi)
    ctx, _, off = _built(systems)
    _check(ctx, off, systems)


def test_hilbert_keys_of_one_block(cuda):
    """Hilbert keys: many small systems, sorted by one block each, and the same few
    at a time beside a larger one, sorted by clusters."""
    systems = [ic.plummer(k, seed=500 + j) for j, k in enumerate(SMALL)]
    ctx, _, off = _built(systems, key_order=1)
    keys, perm = ctx.export_keys()
    for a in range(0, len(systems), 20):
        part = systems[a:a + 20] + [ic.plummer(1000, seed=1)]
        c, _, o = _built(part, key_order=1)
        k, p = c.export_keys()
        n = o[20]
        assert np.array_equal(keys[off[a]:off[a] + n], k[:n])
        assert np.array_equal(perm[off[a]:off[a] + n] - off[a], p[:n])


def test_a_build_of_many_tiny_systems(cuda):
    """2^17 systems of eight bodies build in at most six times the time of one
    system of 2^20 (a cluster of four blocks per system, and boxes that one block
    finished for all of them, took more than eleven times as long)."""
    import torch
    from nns_gb300.barnes_hut import Context, State
    b = ic.plummer(1 << 20, seed=9)
    s = State.from_bodies(b)
    best = []
    for sizes in (1, 1 << 17):
        ctx = Context(max_bodies=1 << 20, max_systems=sizes)
        ctx.set_systems(np.arange(sizes + 1) * ((1 << 20) // sizes))
        t = []
        for _ in range(12):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            ctx.build(s)
            e1.record()
            e1.synchronize()
            t.append(e0.elapsed_time(e1))
        ctx.sync()
        best.append(min(t))
    assert best[1] <= 6 * best[0], best


# merging up to 2^19 bodies a system, and in batches by their sum (2^21; 3 x 2^20 where
# one launch merges; any where it merges four runs); else radix: one-sweep passes below
# 1.5 x 2^20 bodies outside a captured graph, else scanned ones.  Systems of one radix
# tile and of several, in one batch.
SORTS = {
    "merge-top": [524288],
    "sweep": [524289],
    "sweep-batch": [1, 300, 524289, 5000, 2],
    "scan-batch": [1, 300, 524289, 5000, 1100000, 31],
    "merge-two": [16385] * 127,
    "scan-two": [16385] * 129,
    "merge-one": [16384] * 191,
    "scan-one": [16384] * 193,
    "merge-four": [4096] * 800,
    "scan-five": [4097] * 768 + [1],
}


@pytest.mark.parametrize("name", list(SORTS))
def test_both_sides_of_the_sort_rule(cuda, name):
    from nns_gb300.barnes_hut import Context, State
    sizes = SORTS[name]
    n = sum(sizes)
    whole = ic.plummer(n, seed=17)  # any stretch of it is a system of its own box
    off = np.concatenate([[0], np.cumsum(sizes)])
    want_k, want_p = np.empty(n, np.uint64), np.empty(n, np.int32)
    for a, e in zip(off[:-1], off[1:]):
        x, y, z = (np.ascontiguousarray(v[a:e]) for v in (whole.x, whole.y, whole.z))
        hi, lo = O.keys(x, y, z, O.bbox(x, y, z), 42)
        o = np.lexsort((lo, hi))
        want_k[a:e], want_p[a:e] = hi[o], o + a
    ctx = Context(max_bodies=n, max_systems=len(sizes), theta=1.0, eps=0.1)
    ctx.set_systems(off)
    for bits in (8, 9):
        for captured in (False, True):
            ctx.set_tuning(bits, 512)
            s = State.from_bodies(whole)
            if captured:
                ctx.graph_step(s, 1)
            else:
                ctx.build(s)
            ctx.sync()
            keys, perm = ctx.export_keys()
            assert np.array_equal(perm, want_p), (bits, captured)
            assert np.array_equal(keys, want_k), (bits, captured)
