"""The list builder where its groups, rounds and rows end: cells of 1 to 80
atoms (several groups of 16 per cell), empty cells, candidates that fill a
staging round exactly, rows that overflow and grow, and rows so long that a
group takes fewer atoms.  Pairs and their order are the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lists(rows):
    """The rows by atom, each atom's in their order."""
    rows = np.asarray(rows, dtype=np.int64).reshape(-1, 5)
    return rows[np.argsort(rows[:, 0], kind="stable")]


def _check(gpu, oracle, pos, hi, rc, skin):
    lo = np.zeros(3)
    x, y, z = (np.ascontiguousarray(pos[:, k]) for k in range(3))
    ids = np.arange(len(x), dtype=np.uint64)
    ref = _lists(oracle.build_neighbors(x, y, z, ids, lo, hi, rc + skin).pairs_with_ids(ids))
    with gpu.Context(0) as ctx:
        ctx.set_box(lo, hi)
        ctx.set_species([1.0])
        ctx.upload(x, y, z)
        ctx.set_lj(1.0, 0.1, rc)
        ctx.set_skin(skin)
        ctx.build_neighbors()
        assert np.array_equal(_lists(ctx.export_pairs()), ref)
        ctx.build_neighbors()  # from the sorted state
        assert np.array_equal(_lists(ctx.export_pairs()), ref)


@pytest.mark.parametrize("per_cell", [1, 2, 15, 16, 17, 31, 32, 33, 49, 80])
def test_cells_of_every_fill(gpu, oracle, per_cell):
    rng = np.random.default_rng(per_cell)
    edge, k = 1.0, 4
    cell = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = ((cell[:, None, :] + rng.uniform(0.02, 0.98, (len(cell), per_cell, 3))) * edge).reshape(-1, 3)
    _check(gpu, oracle, pos, np.full(3, k * edge), 0.9, 0.09)


@pytest.mark.parametrize("n", [1, 2, 37, 700])
def test_empty_cells_and_clusters(gpu, oracle, n):
    """A dense cluster in a mostly empty box: empty stencil cells, rows far
    above the first capacity estimate (overflow, regrow)."""
    rng = np.random.default_rng(n)
    pos = np.mod(rng.normal(0.0, 0.35, (n, 3)), 9.0)
    pos[pos >= 9.0] = 0.0
    _check(gpu, oracle, pos, np.full(3, 9.0), 1.2, 0.3)


def test_rows_beyond_a_warps_shared_memory(gpu, oracle):
    """About 4,000 neighbours per atom: groups of fewer than 16 atoms."""
    rng = np.random.default_rng(5)
    pos = np.mod(rng.normal(0.0, 0.2, (4_200, 3)), 6.0)
    pos[pos >= 6.0] = 0.0
    _check(gpu, oracle, pos, np.full(3, 6.0), 1.4, 0.1)
