"""Forces, energies and virials at the launch the library picks for the number
of atoms (lanes per atom, block): the sizes on both sides of each change, odd
atom counts (blocks and warps that end short), list rows of every remainder,
against the FP64 oracle.  A filtered (two-level) list must hold the same pairs
as a fresh one in every layout."""
import numpy as np
import pytest

from exastamp_gb300 import setfl as SF
from exastamp_gb300 import systems as S

pytestmark = pytest.mark.gpu


def _atoms(n, a, seed, disp):
    k = int(np.ceil((n / 4.0) ** (1.0 / 3.0)))
    pos, lo, hi = S.lattice(k, k, k, a, S.FCC_BASIS)
    rng = np.random.default_rng(seed)
    pos = pos[np.sort(rng.permutation(len(pos))[:n])]  # vacancies down to n
    pos = np.mod(pos + rng.normal(0.0, disp, pos.shape), hi)
    pos[pos >= hi] = 0.0
    return [np.ascontiguousarray(pos[:, d]) for d in range(3)], lo, hi, rng


def _rel(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


@pytest.mark.parametrize("pot", ["lj", "eam", "alloy"])
@pytest.mark.parametrize("n", [109, 8192, 8193, 24577, 49153])
def test_default_launch_matches_oracle(gpu, oracle, pot, n):
    (x, y, z), lo, hi, rng = _atoms(n, 1.6796 if pot == "lj" else 3.615, n, 0.05)
    ids = np.arange(n, dtype=np.uint64)
    types = (rng.random(n) < 0.5).astype(np.uint8) if pot == "alloy" else np.zeros(n, np.uint8)
    if pot == "lj":
        masses, R = np.array([1.0]), 2.8
        nl = oracle.build_neighbors(x, y, z, ids, lo, hi, R)
        ref = oracle.lj_force(x, y, z, nl, hi - lo, 1.0, 1.0, 2.5)
    else:
        cfg = SF.load_cu_params()
        sf = SF.tabulate(cfg)
        masses, R = sf.masses, 5.3
        if pot == "alloy":
            b = SF.tabulate(cfg, {"A": cfg["params"]["A"] * 1.1, "re": cfg["params"]["re"] * 1.03})
            masses = np.array([sf.masses[0], 1.1 * sf.masses[0]])
            sf = SF.Setfl(["Cu", "Xx"], [29, 30], list(masses), [3.615, 3.615], ["fcc", "fcc"], sf.nrho, sf.drho,
                          sf.nr, sf.dr, sf.rcut, [sf.frho[0], b.frho[0]], [sf.rhor[0], b.rhor[0]],
                          [sf.z2r[0], 0.5 * (sf.z2r[0] + b.z2r[0]), b.z2r[0]])
        tab = oracle.EamOracleTables.from_setfl(sf, S.EV, S.EV, rcut=5.0)
        nl = oracle.build_neighbors(x, y, z, ids, lo, hi, R)
        ref = oracle.eam_forces(x, y, z, types, nl, hi - lo, tab, 5.0)
    F = np.stack(ref[:3], 1) / np.asarray(masses)[types][:, None]
    with gpu.Context(0) as ctx:
        ctx.set_box(lo, hi)
        ctx.set_species(list(masses))
        ctx.upload(x, y, z, types=types)
        if pot == "lj":
            ctx.set_lj(1.0, 1.0, 2.5)
        else:
            ctx.set_eam_alloy(sf, 5.0, S.EV, S.EV)
        ctx.set_skin(0.3)
        assert ctx.get_launch_ex() == (1, 4, 256)  # a pick is not a setting
        for mixed, tol, etol in ((False, 1e-12, 1e-12), (True, 1e-5, 1e-6)):
            ctx.set_precision(mixed)
            ctx.compute_forces(energy=False)
            d = ctx.download(("ax", "ay", "az"))
            assert _rel(np.stack([d["ax"], d["ay"], d["az"]], 1), F) < tol
            ctx.compute_forces(energy=True, virial=True)
            d = ctx.download(("ax", "ay", "az", "ep"), virial=True)
            assert _rel(np.stack([d["ax"], d["ay"], d["az"]], 1), F) < tol
            assert _rel(d["ep"], ref[3]) < 10 * etol
            assert _rel(d["vir"].reshape(n, 9), np.asarray(ref[4]).reshape(n, 9)) < 10 * tol


@pytest.mark.parametrize("tpa,vec", [(0, 0), (1, 4), (2, 4), (4, 4), (4, 1)])
def test_filtered_list_in_every_layout(gpu, tpa, vec):
    s = S.lj_fcc(ncell=8, T=0.1, seed=21)
    pairs = []
    for filtered in (True, False):
        with gpu.Context(0) as ctx:
            if filtered:
                ctx.upload_system(s)
            else:
                ctx.set_box(s.lo, s.hi)
                ctx.set_species([1.0])
                ctx.upload(d["x"], d["y"], d["z"])  # noqa: F821 (set by the first turn)
            ctx.set_lj(1.0, 1.0, 2.5)
            ctx.set_skin(0.3)
            ctx.set_precision(True)
            if filtered:
                ctx.set_list_buffer(1.0)
                if tpa:
                    ctx.set_launch(tpa, 128, vec)
                ctx.run_nve(10, 0.005, rebuild_every=10)
                assert ctx.list_buffer()[1] == 1  # the list came from the filter
                d = ctx.download(("x", "y", "z"))
            # by caller index and without images, which the wrap changes
            pairs.append({(int(r[0]), int(r[1])) for r in ctx.export_pairs()})
            assert filtered or len(pairs[0]) > 100_000
    ids = np.asarray(s.id, dtype=np.int64)
    assert {(int(ids[i]), int(ids[j])) for i, j in pairs[1]} == pairs[0]
