"""Several entries of one list row on the cutoff's edge at once (the LJ kernels
take a row's exact tests behind one branch): the crystal whose fourth shell
sits at rcut gives every atom twelve, spread over its rows in every layout,
with and without energies and virials, against the FP64 oracle."""
import numpy as np
import pytest

from exastamp_gb300 import systems as S

pytestmark = pytest.mark.gpu

RC = 2.5


@pytest.mark.parametrize("multi", [False, True])
@pytest.mark.parametrize("tpa,vec", [(0, 0), (1, 1), (1, 4), (2, 4), (4, 4), (8, 1)])
def test_rows_with_several_edge_pairs(gpu, oracle, tpa, vec, multi):
    a = RC / np.sqrt(2.0)
    pos, lo, hi = S.lattice(5, 4, 3, a, S.FCC_BASIS)
    rng = np.random.default_rng(7)
    pos = np.mod(pos + 0.3 * a + rng.normal(0.0, 1e-6, pos.shape), hi)[:-3]  # a last warp that ends short
    n = len(pos)
    x, y, z = (np.ascontiguousarray(pos[:, k]) for k in range(3))
    nl = oracle.build_neighbors(x, y, z, np.arange(n, dtype=np.uint64), lo, hi, RC + 0.3)
    ref = oracle.lj_force(x, y, z, nl, hi - lo, 1.0, 1.0, RC)
    F, trace = np.stack(ref[:3], 1), np.asarray(ref[4]).reshape(n, 9)[:, [0, 4, 8]].sum(1)
    with gpu.Context(0) as ctx:
        ctx.set_box(lo, hi)
        ctx.set_species([1.0])
        ctx.upload(x, y, z)
        if multi:
            ctx.set_lj_multi(np.array([[1.0]]), np.array([[1.0]]), np.array([[RC]]), RC + 0.5)
            ctx.set_skin(0.0)
        else:
            ctx.set_lj(1.0, 1.0, RC)
            ctx.set_skin(0.3)
        ctx.set_precision(True)
        if tpa:
            ctx.set_launch(tpa, 128, vec)
        # separations to ~3e-7 with force slopes of at most ~60 over 54 pairs
        # are below 1e-3 in a force and in the trace of a virial; a pair on the
        # wrong side is at least 0.0225 in a force and 0.048 in the trace
        ctx.compute_forces(energy=False)
        d = ctx.download(("ax", "ay", "az"))
        assert np.abs(np.stack([d["ax"], d["ay"], d["az"]], 1) - F).max() < 2e-3
        ctx.compute_forces(energy=True, virial=True)
        d = ctx.download(("ax", "ay", "az"), virial=True)
        assert np.abs(np.stack([d["ax"], d["ay"], d["az"]], 1) - F).max() < 2e-3
        assert np.abs(d["vir"].reshape(n, 9)[:, [0, 4, 8]].sum(1) - trace).max() < 5e-3
