"""The autotuner on knobs that do nothing (small systems are walked by teams of fixed
shape and sorted by merging): timings that differ by noise leave the defaults, and
results of other kernels are not reused.  On the CPU, with a fake context and timer.
"""
import json
from types import SimpleNamespace

import numpy as np
import pytest

from nns_gb300 import autotune


class Ctx:
    device = 0

    def __init__(self):
        self.offsets = np.array([0, 4096])
        self.params = SimpleNamespace(compensated=0, radix_bits=8, stack_depth=512, leaf_size=1, key_order=0,
                                      moments_mode=0, multipole=0)
        self.walk = (8, 3)

    def set_walk(self, warps, variant):
        self.walk = (warps, variant)

    def set_tuning(self, bits, depth):
        self.params.radix_bits, self.params.stack_depth = bits, depth

    def build(self, state):
        pass

    forces = build

    def sync(self):
        pass


def _noise(seed, amount):
    rng = np.random.default_rng(seed)
    return lambda fn, reps: 1.0 + amount * float(rng.uniform(-1.0, 1.0))


@pytest.mark.parametrize("seed", range(20))
def test_noise_leaves_the_defaults(monkeypatch, seed):
    monkeypatch.setattr(autotune.torch.cuda, "get_device_name", lambda dev: "fake")
    ctx = Ctx()
    r = autotune.tune_walk(ctx, None, use_cache=False, timer=_noise(seed, 0.45 * autotune.MARGIN))
    assert (ctx.walk, ctx.params.stack_depth, ctx.params.radix_bits) == ((8, 3), 512, 8)
    assert (r["warps"], r["variant"], r["stack_depth"], r["radix_bits"]) == (8, 3, 512, 8)


def test_results_of_other_kernels_are_not_reused(monkeypatch, tmp_path):
    monkeypatch.setattr(autotune.torch.cuda, "get_device_name", lambda dev: "fake")
    monkeypatch.setenv("NBX_AUTOTUNE_CACHE", str(tmp_path / "tune.json"))
    old = {"warps": 16, "variant": 1, "stack_depth": 768, "radix_bits": 9}
    key = "fake|n=4096|sys=1|comp=0|order=0|moments=0|multipole=0"
    (tmp_path / "tune.json").write_text(json.dumps({key: old}))
    ctx = Ctx()
    assert not autotune.tune_walk(ctx, None, timer=_noise(1, 0.0))["cached"]
    assert ctx.walk == (8, 3)
    assert autotune.tune_walk(Ctx(), None, timer=lambda fn, reps: pytest.fail("timed a cached entry"))["cached"]
