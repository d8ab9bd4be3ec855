"""Pair membership in cells far wider than the list radius: an axis holds at most
1,024 cells, so in a long thin box they grow with the box, and with them the
rounding of the FP32 cell-relative positions.  A slab of an FCC crystal, its
fourth shell on the cutoff and its fifth on the list radius, sits at the far
end of a cell 400 radii wide.  The pair list, and the forces, which jump at the
cutoff, against the FP64 oracle in both precisions."""
import numpy as np
import pytest

from exastamp_gb300 import systems as S

pytestmark = pytest.mark.gpu

RC = 2.5
A = RC / np.sqrt(2.0)
SKIN = A * np.sqrt(2.5) - RC


def _slab(axis):
    n = [3, 3, 3]
    n[axis] = 12
    pos, lo, hi = S.lattice(n[0], n[1], n[2], A, S.FCC_BASIS)
    rng = np.random.default_rng(17 + axis)
    pos = np.mod(pos + 0.3 * A + rng.normal(0.0, 1e-5, pos.shape), hi)
    h = 400.0 * (RC + SKIN)
    hi = hi.copy()
    hi[axis] = 1024.0 * h
    pos[:, axis] += 0.9 * h
    return [np.ascontiguousarray(pos[:, d]) for d in range(3)], lo, hi


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("multi", [False, True])
@pytest.mark.parametrize("axis", [0, 2])
def test_membership_in_wide_cells_is_that_of_fp64(gpu, oracle, axis, multi, mixed):
    (x, y, z), lo, hi = _slab(axis)
    ids = np.arange(len(x), dtype=np.uint64)
    nl = oracle.build_neighbors(x, y, z, ids, lo, hi, RC + SKIN)
    ref = np.stack(oracle.lj_force(x, y, z, nl, hi - lo, 1.0, 1.0, RC, virial=False)[:3], 1)
    with gpu.Context(0) as ctx:
        ctx.set_box(lo, hi)
        ctx.set_species([1.0])
        ctx.upload(x, y, z)
        if multi:
            ctx.set_lj_multi(np.array([[1.0]]), np.array([[1.0]]), np.array([[RC]]), RC + SKIN)
            ctx.set_skin(0.0)
        else:
            ctx.set_lj(1.0, 1.0, RC)
            ctx.set_skin(SKIN)
        ctx.set_precision(mixed)
        for launch in ((0, 0), (1, 1), (4, 4)):
            if launch[0]:
                ctx.set_launch(launch[0], 128, launch[1])
            assert len(ctx.export_pairs()) == len(nl.nbr)
            ctx.compute_forces(energy=False)
            d = ctx.download(("ax", "ay", "az"))
            got = np.stack([d["ax"], d["ay"], d["az"]], 1)
            # FP64: rounding.  Mixed: two coordinates below 1,024, each off by at
            # most 2^-15, put a separation off by at most 1.06e-4; the pair
            # stiffnesses of the shells (12 x 1.9, 6 x 1.55, 24 x 0.34, 12 x 0.11)
            # sum to 41.5: at most 4.4e-3.  A pair on the wrong side is at
            # least 0.039 / sqrt(3) = 0.0225.
            assert np.abs(got - ref).max() < (6e-3 if mixed else 1e-10)
