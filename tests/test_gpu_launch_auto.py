"""The launch in effect: what the library picks on both sides of its atom-count
thresholds, and the way back to it after a launch was set."""
import numpy as np
import pytest

from exastamp_gb300 import systems as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,lanes", [(8192, 16), (8193, 8), (24576, 8), (24577, 4), (49153, 2), (262145, 1)])
def test_automatic_launch_comes_back(gpu, n, lanes):
    k = int(np.ceil((n / 4.0) ** (1.0 / 3.0)))
    pos, lo, hi = S.lattice(k, k, k, 1.6796, S.FCC_BASIS)
    pos = pos[:n]
    with gpu.Context(0) as ctx:
        ctx.set_box(lo, hi)
        ctx.set_species([1.0])
        ctx.upload(*(np.ascontiguousarray(pos[:, d]) for d in range(3)))
        ctx.set_lj(1.0, 1.0, 2.5)
        ctx.set_skin(0.3)
        ctx.compute_forces(energy=False)
        picked = ctx.get_launch_used()
        assert picked == (lanes, 4, 256 if lanes == 1 else 128) and ctx.get_launch_ex() == (1, 4, 256)
        a = ctx.download(("ax", "ay", "az"))
        ctx.set_launch(4, 64, 1)
        ctx.compute_forces(energy=False)
        assert ctx.get_launch_used() == ctx.get_launch_ex() == (4, 1, 64)
        ctx.set_launch_auto()
        ctx.compute_forces(energy=False)
        assert ctx.get_launch_used() == picked and ctx.get_launch_ex() == (1, 4, 256)
        b = ctx.download(("ax", "ay", "az"))
        assert all(np.array_equal(a[q], b[q]) for q in a)
