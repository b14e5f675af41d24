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
