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


def _rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return np.linalg.norm(a - b, axis=1) / np.maximum(np.linalg.norm(b, axis=1), 1e-30)


def _walk(b, variant=3, warps=8, eps=0.01, **kw):
    from nns_gb300.barnes_hut import Context, State
    n = len(b.x)
    ctx = Context(max_bodies=n, theta=0.5, eps=eps, **kw)
    ctx.set_walk(warps, variant)
    ctx.set_systems([0, n])
    s = State.from_bodies(b)
    ctx.build(s)
    ctx.forces(s)
    ctx.sync()
    return ctx, s


BODIES = {"disk20011": lambda: ic.star_disk(20011), "plummer16385": lambda: ic.plummer(16385),
          "binary160033": lambda: ic.binary_disk(160033)}  # the last: more than 32 groups per SM
_cache = {}


def _want(name, leaf, multipole, eps=0.01):
    key = (name, leaf, multipole)
    if key not in _cache:
        b = BODIES[name]()
        t = O.build(b.x, b.y, b.z, b.m)
        q = O.quadrupoles(b.x, b.y, b.z, b.m, t) if multipole else None
        e = np.float32(eps)
        _cache[key] = b, O.forces(b.x, b.y, b.z, b.m, O.bucket_tree(t, leaf) if leaf > 1 else t, 0.25, float(e * e),
                                  quad=q)
    return _cache[key]


@pytest.mark.parametrize("name,leaf,multipole", [("disk20011", 1, 0), ("disk20011", 1, 1), ("disk20011", 4, 0),
                                                 ("disk20011", 4, 1), ("plummer16385", 1, 0), ("plummer16385", 1, 1),
                                                 ("binary160033", 1, 0), ("binary160033", 1, 1)])
@pytest.mark.parametrize("variant", [0, 1, 2, 3])
def test_every_form_matches_oracle(cuda, name, leaf, multipole, variant):
    """The accumulation modes of every variant (the one-cell walk has no quadrupoles)
    on the oracle's lists, within the walk tests' bounds of its FP64 sums."""
    if variant == 2 and multipole:
        pytest.skip("the one-cell walk has monopoles only")
    b, f = _want(name, leaf, multipole)
    for comp in (0, 1, 2):
        ctx, s = _walk(b, variant, leaf_size=leaf, multipole=multipole, compensated=comp)
        nl, no = ctx.walk_stats()
        assert np.array_equal(nl, f.nlist) and np.array_equal(no, f.nopen), comp
        rel = _rel(s.acc(), f.a64)
        assert np.median(rel) <= MED_TOL and rel.max() <= MAX_TOL, (comp, np.median(rel), rel.max())


@pytest.mark.parametrize("n", [20011, 160033])
@pytest.mark.parametrize("variant", [0, 1, 3])
@pytest.mark.parametrize("multipole", [0, 1])
def test_launch_shapes_agree(cuda, n, variant, multipole):
    """Blocks of two warps (a launch that fits the GPU at once) and of the asked 4, 8
    and 16: the same bits."""
    b = ic.plummer(n)
    out = [_walk(b, variant, warps, multipole=multipole)[1].acc() for warps in (4, 8, 16)]
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


def test_potential(cuda):
    b = ic.plummer(20011)
    ctx, s = _walk(b)
    phi = ctx.potential(s)
    e = np.float32(0.01)
    tg = np.arange(0, 20011, 7)
    want = O.direct_potential_fp64(b.x, b.y, b.z, b.m, float(e * e), tg)
    rel = np.abs(phi[tg] - want) / np.abs(want)
    assert np.median(rel) < 1e-3 and rel.max() < 2e-2  # the monopole potential's bounds of the parity tests


@pytest.mark.parametrize("name", ["collinear", "coplanar", "signed_zeros", "cluster", "deep"])
@pytest.mark.parametrize("variant", [0, 1, 3])
@pytest.mark.parametrize("multipole", [0, 1])
def test_adversarial_geometry(cuda, name, variant, multipole):
    """The adversarial sets with enough bodies for the walk by single warps: lists
    bit-exact, each body's error bounded relative to its own force plus the set's
    median force (pulls that nearly cancel on a line or in a plane)."""
    from adversarial import CASES, EPS
    key = (name, multipole)
    eps = EPS.get(name, 0.01)
    if key not in _cache:
        b = CASES[name](24000)
        assert len(b.x) > 1 << 14
        t = O.build(b.x, b.y, b.z, b.m)
        q = O.quadrupoles(b.x, b.y, b.z, b.m, t) if multipole else None
        e = np.float32(eps)
        _cache[key] = b, O.forces(b.x, b.y, b.z, b.m, t, 0.25, float(e * e), quad=q)
    b, f = _cache[key]
    ctx, s = _walk(b, variant, eps=eps, multipole=multipole)
    nl, no = ctx.walk_stats()
    assert np.array_equal(nl, f.nlist) and np.array_equal(no, f.nopen)
    a = s.acc().astype(np.float64)
    err, mag = np.linalg.norm(a - f.a64, axis=1), np.linalg.norm(f.a64, axis=1)
    assert np.median(_rel(a, f.a64)) <= MED_TOL
    assert (err <= MAX_TOL * (mag + np.median(mag))).all(), (err / (mag + np.median(mag))).max()


def test_the_adjoint_records_this_walk(cuda):
    """The trajectory gradients of a system above the teams' size: the forward ends bit
    for bit where ordinary steps end, and the gradients agree with FP64 central
    finite differences of the FP64 replay (bound of the adjoint tests)."""
    import torch
    from nns_gb300.adjoint import Adjoint, random_directions
    from nns_gb300.barnes_hut import Context, State
    n, T = 20011, 5
    b = ic.plummer(n, seed=ic.SEED0 + 3)
    ctx = Context(max_bodies=n, theta=0.5, eps=0.01, dt=1e-3)
    ctx.set_systems([0, n])
    s = State.from_bodies(b)
    ctx.step(s, T)
    ctx.sync()
    end = s.host()
    noise = 0.01 * np.random.default_rng(3).standard_normal((3, n))
    target = torch.as_tensor((np.stack(end[:3]) + noise).astype(np.float32), device="cuda")
    adj = Adjoint(ctx, T, 2, 8192, T)
    r = State.from_bodies(b)
    loss32 = adj.forward(r, target)
    for got, want in zip(r.host(), end):
        assert np.array_equal(got, want)
    g = np.concatenate([t.cpu().numpy().reshape(-1, n) for t in adj.backward(r)]).astype(np.float64)
    adj.record(State.from_bodies(b))
    base = np.stack([b.x, b.y, b.z, b.vx, b.vy, b.vz, b.m]).astype(np.float64)
    dev = lambda a: torch.as_tensor(a, device="cuda")  # noqa: E731
    assert abs(adj.replay_fp64(dev(base)) - loss32) / loss32 < 1e-4
    h, gnorm = 1e-6, np.linalg.norm(g)
    for u in random_directions(n, 4):
        fd = (adj.replay_fp64(dev(base + h * u)) - adj.replay_fp64(dev(base - h * u))) / (2 * h)
        assert abs(fd - float((g * u).sum())) <= 1e-4 * gnorm


@pytest.mark.parametrize("n", [4000, 20011, 60000])
@pytest.mark.parametrize("stack_depth", [360, 384, 512])
@pytest.mark.parametrize("kw", [{}, {"compensated": 1}, {"multipole": 1}], ids=["plain", "split", "quad"])
def test_small_opening_angles_fill_the_stack(cuda, n, stack_depth, kw):
    """theta = 0.1375 opens most cells, so the stack fills to its depth-first reserve and
    rounds pop what room is left: the oracle's lists with any stack, and never more
    than two and a half times the rounds of a stack that always has room (one cell a
    round near the reserve took ten times as many)."""
    from nns_gb300.barnes_hut import Context, State
    key = ("theta", n, kw.get("multipole", 0))
    e = np.float32(0.005)
    if key not in _cache:
        b = ic.plummer(n)
        t = O.build(b.x, b.y, b.z, b.m)
        q = O.quadrupoles(b.x, b.y, b.z, b.m, t) if key[2] else None
        th = np.float32(0.1375)
        _cache[key] = b, O.forces(b.x, b.y, b.z, b.m, t, float(th * th), float(e * e), quad=q)
    b, f = _cache[key]
    rounds = []
    for depth in (stack_depth, 2048):
        ctx = Context(max_bodies=n, theta=0.1375, eps=0.005, stack_depth=depth, **kw)
        ctx.set_systems([0, n])
        s = State.from_bodies(b)
        ctx.build(s)
        ctx.forces(s)
        ctx.sync()
        nl, no = ctx.walk_stats()
        assert np.array_equal(nl, f.nlist) and np.array_equal(no, f.nopen)
        rel = _rel(s.acc(), f.a64)
        assert np.median(rel) <= MED_TOL and rel.max() <= MAX_TOL, depth
        rounds.append(ctx.tree_info()["rounds"])
    assert rounds[0] <= 2.5 * rounds[1], rounds


@pytest.mark.parametrize("name", ["star_disk", "binary_disk", "plummer"])
@pytest.mark.parametrize("n,bound", [(5003, 2.5e-7), (16384, 2.5e-7), (131071, 3.5e-7)])
def test_plain_sums_keep_their_precision(cuda, name, n, bound):
    """The plain FP32 sums against FP64 sums of the same lists.  Every body's rounding
    is that of its own round's terms and one sum per round: with about 20 rounds of
    64 adds in two halves, r.m.s. below 2^-24 sqrt(20 + 32) = 4.3e-7, as the largest
    term is rarely most of the force below 3.5e-7, by teams (four sums, 10 rounds of
    up to 48) below 2.5e-7.  (One running sum had 0.7e-6 to 2.2e-6 on the disks.)"""
    from nns_gb300.barnes_hut import Context, State
    b = getattr(ic, name)(n)
    ctx, s = _walk(b)
    tg = np.arange(0, n, max(1, n // 8000))
    a, w = s.acc()[tg].astype(np.float64), ctx.forces_fp64_lists(tg)
    e = _rel(a, w)
    assert np.sqrt(np.mean(e * e)) <= bound


@pytest.mark.parametrize("warps", [4, 8, 16])
@pytest.mark.parametrize("stack_depth", [1824, 1940, 2016])
def test_deep_stacks_fit_as_before(cuda, warps, stack_depth):
    """Stacks that just fitted a launch shape before the rounds' totals took shared
    memory of their own go out in smaller blocks, with the same bits."""
    from nns_gb300.barnes_hut import Context, State
    b = ic.plummer(160033)
    acc = []
    for w in (warps, 4):
        ctx = Context(max_bodies=len(b.x), theta=0.5, eps=0.01, multipole=1, stack_depth=stack_depth)
        ctx.set_walk(w, 3)
        ctx.set_systems([0, len(b.x)])
        s = State.from_bodies(b)
        ctx.build(s)
        ctx.forces(s)
        ctx.sync()
        acc.append(s.acc())
    assert np.array_equal(acc[0], acc[1])
