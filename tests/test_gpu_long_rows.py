"""Neighbour lists with long rows, which another kernel builds: capacities on both
sides of its threshold of 900 entries, full and half lists, against the oracle's
pairs; its gated form in a run with the displacement trigger; and rows of more
than 40,000 entries, once refused, against a count in FP64."""
import numpy as np
import pytest

from exastamp_gb300 import systems as S

pytestmark = pytest.mark.gpu


def _crystal(k, a, seed):
    pos, lo, hi = S.lattice(k, k, k, a, S.FCC_BASIS)
    pos = np.mod(pos + np.random.default_rng(seed).normal(0.0, 0.05 * a, pos.shape), hi)
    pos[pos >= hi] = 0.0
    return [np.ascontiguousarray(pos[:, d]) for d in range(3)], lo, hi


@pytest.mark.parametrize("R,capacity", [(5.6, 896), (5.8, 960)])
@pytest.mark.parametrize("half", [False, True])
def test_pairs_on_both_sides_of_the_threshold(gpu, oracle, R, capacity, half):
    (x, y, z), lo, hi = _crystal(8, 1.6796, 3)
    n = len(x)
    ids = np.arange(n, dtype=np.uint64)
    nl = oracle.build_neighbors(x, y, z, ids, lo, hi, R)
    with gpu.Context(0) as ctx:
        ctx.set_box(lo, hi)
        ctx.set_species([1.0])
        ctx.upload(x, y, z)
        ctx.set_lj(1.0, 1.0, 2.5)
        ctx.set_skin(R - 2.5)
        ctx.set_precision(True)
        ctx.set_newton3(half)
        ctx.build_neighbors()
        assert half or ctx.neighbor_stats()[1] == capacity
        got = {tuple(int(v) for v in r) for r in ctx.export_pairs()}
    ref = {tuple(int(v) for v in r) for r in nl.pairs_with_ids(ids)}
    if half:  # each unordered pair once
        other = {(j, i, -a, -b, -c) for i, j, a, b, c in got}
        assert not got & other
        got |= other
    assert got == ref


def test_trigger_rebuilds_long_rows(gpu, oracle):
    (x, y, z), lo, hi = _crystal(8, 1.6796, 4)
    n = len(x)
    v = np.random.default_rng(5).normal(0.0, 2.0, (3, n))
    with gpu.Context(0) as ctx:
        ctx.set_box(lo, hi)
        ctx.set_species([1.0])
        ctx.upload(x, y, z, *v)
        ctx.set_lj(1.0, 1.0, 5.5)
        ctx.set_skin(0.3)
        ctx.set_precision(False)
        for graph in (False, True):
            before = ctx.list_builds()
            ctx.run_nve(40, 0.002, rebuild_every=-1, use_graph=graph)
            assert ctx.neighbor_stats()[1] >= 900 and ctx.list_builds() > before
            d = ctx.download(("x", "y", "z", "ax", "ay", "az"))
            w = [np.mod(d[k], hi[q]) for q, k in enumerate("xyz")]
            nl = oracle.build_neighbors(*w, np.arange(n, dtype=np.uint64), lo, hi, 5.8)
            ref = np.stack(oracle.lj_force(*w, nl, hi - lo, 1.0, 1.0, 5.5, virial=False)[:3], 1)
            got = np.stack([d["ax"], d["ay"], d["az"]], 1)
            # FP64 with positions wrapped in another order: 1e-13 relative, and
            # no pair within that of the cutoff
            assert np.sqrt(((got - ref) ** 2).sum() / (ref ** 2).sum()) < 1e-11


def test_rows_beyond_shared_memory(gpu):
    import torch

    (x, y, z), lo, hi = _crystal(14, 10.0 / 14, 6)
    n, R = len(x), 9.99
    with gpu.Context(0) as ctx:
        ctx.set_box(lo, hi)
        ctx.set_species([1.0])
        ctx.upload(x, y, z)
        ctx.set_lj(1.0, 0.3, 0.75)
        ctx.set_precision(False)
        a = []
        for skin in (0.1, R - 0.75):
            ctx.set_skin(skin)
            ctx.compute_forces(energy=False)
            d = ctx.download(("ax", "ay", "az"))
            a.append(np.stack([d["ax"], d["ay"], d["az"]], 1))
        npairs, capacity, _ = ctx.neighbor_stats()
    assert capacity > 51_000
    # the same pairs within the cutoff, summed in another order
    assert np.sqrt(((a[1] - a[0]) ** 2).sum() / (a[0] ** 2).sum()) < 1e-13
    p = torch.tensor(np.stack([x, y, z]), device="cuda")
    L = torch.tensor(hi - lo, device="cuda")
    total = 0
    for s in range(27):
        image = torch.tensor([s % 3 - 1, s // 3 % 3 - 1, s // 9 - 1], device="cuda") * L
        for i0 in range(0, n, 1024):
            d2 = 0.0
            for k in range(3):  # x, y, z in turn, each operation rounded
                dk = (p[k] + image[k])[None, :] - p[k, i0:i0 + 1024, None]
                d2 = d2 + dk * dk
            total += int((d2 <= R * R).sum())
    assert npairs == total - n  # without the atoms themselves
