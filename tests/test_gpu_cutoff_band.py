"""Cutoff membership of the mixed kernels at distances that FP32 cannot tell
apart from the cutoff: an FCC crystal whose fourth shell sits at rcut, shaken
by 1e-7 to 1e-3, so that every atom has twelve pairs on the edge.  The LJ force
jumps by 0.039 there, so one pair on the wrong side is an error far above the
tolerance."""
import numpy as np
import pytest

from exastamp_gb300 import systems as S

pytestmark = pytest.mark.gpu

RC = 2.5


@pytest.mark.parametrize("ncell", [2, 3, 8])
@pytest.mark.parametrize("shake", [1e-7, 3e-6, 1e-4, 1e-3])
@pytest.mark.parametrize("multi", [False, True])
def test_membership_at_the_cutoff_is_that_of_fp64(gpu, oracle, ncell, shake, multi):
    a = RC / np.sqrt(2.0)
    pos, lo, hi = S.lattice(ncell, ncell, ncell, a, S.FCC_BASIS)
    rng = np.random.default_rng(int(ncell * 1e8 * shake) + 5)
    pos = np.mod(pos + 0.3 * a + rng.normal(0.0, shake, pos.shape), hi)
    x, y, z = (np.ascontiguousarray(pos[:, k]) for k in range(3))
    ids = np.arange(len(x), dtype=np.uint64)
    nl = oracle.build_neighbors(x, y, z, ids, lo, hi, RC + 0.3)
    ref = np.stack(oracle.lj_force(x, y, z, nl, hi - lo, 1.0, 1.0, RC, virial=False)[:3], 1)
    with gpu.Context(0) as ctx:
        ctx.set_box(lo, hi)
        ctx.set_species([1.0])
        ctx.upload(x, y, z)
        if multi:  # a list reaching far beyond this pair's cutoff
            ctx.set_lj_multi(np.array([[1.0]]), np.array([[1.0]]), np.array([[RC]]), RC + 0.5)
            ctx.set_skin(0.0)
        else:
            ctx.set_lj(1.0, 1.0, RC)
            ctx.set_skin(0.3)
        ctx.set_precision(True)
        ctx.compute_forces(energy=False)
        d = ctx.download(("ax", "ay", "az"))
    got = np.stack([d["ax"], d["ay"], d["az"]], 1)
    # FP32 pair arithmetic: separations to ~3e-7, pair forces of at most ~3
    # with slopes of at most ~60 over 54 pairs of random sign -> below 2e-4; a pair
    # on the wrong side is at least 0.039 / sqrt(3) = 0.0225
    assert np.abs(got - ref).max() < 2e-3
