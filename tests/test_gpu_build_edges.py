"""Tree build at the sizes where its kernels change shape: block edges of the node
kernels (512 positions), the switch between summed and scanned level counts
(131072 positions) and between the one-block and the cluster form of the top
cells' sums (65536), with the centre-of-mass passes of every mode.  Bit-exact
against the oracle.
"""
import numpy as np
import pytest

from nns_gb300 import ic
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(b, gt, ot):
    assert np.array_equal(gt["perm"], ot.perm)
    assert np.array_equal(gt["root_child"], ot.root_child)
    assert gt["ncells"] == ot.ncells
    for k in ("cell_child", "cell_start", "cell_count", "cell_level", "cell_x", "cell_y", "cell_z", "cell_m"):
        assert np.array_equal(gt[k], getattr(ot, k)), k


@pytest.mark.parametrize("n", [511, 512, 513, 1025, 65536, 65537, 131072, 131073])
@pytest.mark.parametrize("moments_mode", [0, 1, 2])
def test_node_blocks(cuda, n, moments_mode):
    from nns_gb300.barnes_hut import Context, State
    b = ic.plummer(n, seed=n)
    ctx = Context(max_bodies=n, moments_mode=moments_mode)
    ctx.set_systems([0, n])
    ctx.build(State.from_bodies(b))
    ctx.sync()
    _check(b, ctx.export_tree(0), O.build(b.x, b.y, b.z, b.m))


# moments_mode 0 takes one launch up to 2^21 bodies, in batches up to 2^22, and to 2^23
# where no system has more than 2^16; else one launch per level
@pytest.mark.parametrize("sizes", [[1 << 21], [(1 << 21) + 1], [(1 << 21) - 5, (1 << 21) + 5], [1 << 21, (1 << 21) + 1],
                                   [65536] * 65, [65537] * 64 + [100]],
                         ids=["2^21", "2^21+1", "2^22", "2^22+1", "many", "many-larger"])
@pytest.mark.parametrize("multipole", [0, 1])
def test_moments_of_every_mode(cuda, sizes, multipole):
    """The three modes sum the same FP64 additions in the same order: the same forces
    bit for bit, on both sides of the sizes where mode 0 changes its launches."""
    from nns_gb300.barnes_hut import Context, State
    n = sum(sizes)
    b = ic.plummer(n, seed=n)
    got = []
    for mode in (0, 1, 2):
        ctx = Context(max_bodies=n, max_systems=len(sizes), moments_mode=mode, multipole=multipole, theta=1.0, eps=0.1)
        ctx.set_systems(np.concatenate([[0], np.cumsum(sizes)]))
        s = State.from_bodies(b)
        ctx.build(s)
        ctx.forces(s)
        ctx.sync()
        got.append(s.acc())
    assert np.isfinite(got[0]).all()
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
