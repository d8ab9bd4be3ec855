"""The autotuner never leaves a launch behind that is slower than the library's
own choice, which has shapes that cannot be set; and what it cached for other
kernels does not count.  Over stand-ins with made-up timings."""
import json
import time

import pytest

from exastamp_gb300 import autotune


class Ctx:
    """4,000 atoms: the automatic launch (16 lanes x 4) at 13 us, others more."""
    n = 4000

    def __init__(self, auto_us):
        self.launch, self.auto_us, self.density, self.staged = None, auto_us, 128, False

    def set_launch(self, lanes, block, vec=1):
        assert not (vec == 4 and lanes > 4)  # refused by the library
        self.launch = (lanes, vec, block)

    def set_launch_auto(self):
        self.launch = None

    def get_launch_used(self):
        return self.launch or (16, 4, 128)

    def set_density_block(self, block):
        self.density = block

    def get_density_block(self):
        return self.density

    def set_neighbor_staging(self, on):
        self.staged = on

    def profile_step(self, reps=3):
        us = 18.0 + self.launch[0] + (self.launch[1] == 1) + self.launch[2] / 256 if self.launch else self.auto_us
        return {"density": us / 2, "pair": us / 2}


@pytest.mark.parametrize("auto_us,wins", [(13.0, True), (60.0, False)])
def test_tune_keeps_the_automatic_launch_unless_beaten(monkeypatch, tmp_path, auto_us, wins):
    monkeypatch.setenv("GBMD_AUTOTUNE_CACHE", str(tmp_path / "c.json"))
    for _ in range(2):  # measured, then from the cache
        ctx = Ctx(auto_us)
        used = autotune.tune(ctx, "w")[:3]
        assert (ctx.launch is None) == wins and used == ctx.get_launch_used()
        assert ctx.density == (128 if wins else 64) and not ctx.staged
    # other kernels: measured again
    monkeypatch.setattr(autotune, "_kernels", lambda: "others")
    ctx = Ctx(73.0 - auto_us)
    autotune.tune(ctx, "w")
    assert (ctx.launch is None) == (not wins)
    assert len(json.load(open(tmp_path / "c.json"))) == 2


class Batch:
    nrep, n = 256, 256 * 243

    def __init__(self):
        self.small = 0

    def set_launch(self, block, stencil):
        self.shape = (block, stencil)

    def set_small_block(self, block):
        assert 64 <= block <= 256
        self.small = block

    def set_small_block_auto(self):
        self.small = 0

    def run(self, adjoint=False):
        time.sleep(0.002 if self.small else 0.0005)

    def synchronize(self):
        pass


def test_tune_batch_keeps_the_automatic_small_block(monkeypatch, tmp_path):
    monkeypatch.setenv("GBMD_AUTOTUNE_CACHE", str(tmp_path / "c.json"))
    for _ in range(2):
        b = Batch()
        b.small = 128
        assert autotune.tune_batch(b, "w")[2] == 0 and b.small == 0
