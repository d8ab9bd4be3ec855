"""Batched replicas where the lanes per atom, the list builder's groups and the
pair list end: 1 to 2,048 atoms in one launch, every block size, an overflowing
list (evaluated from the cells) with its gradient, and pairs at the cutoff."""
import numpy as np
import pytest

from exastamp_gb300 import setfl as SF
from exastamp_gb300 import systems as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cu():
    cfg = SF.load_cu_params()
    return cfg, SF.tabulate(cfg)


def _cut(s, n):
    pos = np.stack([s.x, s.y, s.z], 1)[:n]
    return S._make(pos, s.lo, s.hi, np.zeros(n), np.array([63.546]), np.zeros_like(pos), {})


def _box(k, a, sig, seed, shift=0.0):
    pos, lo, hi = S.lattice(k, k, k, a, S.FCC_BASIS)
    pos = np.mod(pos + shift + np.random.default_rng(seed).normal(0.0, sig, pos.shape), hi)
    pos[pos >= hi] = 0.0
    return S._make(pos, lo, hi, np.zeros(len(pos)), np.array([63.546]), np.zeros_like(pos), {})


def _forward(oracle, reps, tab):
    F, E = [], []
    for s in reps:
        nl = oracle.build_neighbors(s.x.copy(), s.y.copy(), s.z.copy(), s.id, s.lo, s.hi, 5.0)
        r = oracle.eam_forces(s.x, s.y, s.z, s.type, nl, s.L, tab, 5.0)
        F.append(np.stack(r[:3], 1))
        E.append(r[3])
    return np.concatenate(F), np.concatenate(E)


@pytest.mark.parametrize("small,big", [(0, 0), (64, 64), (96, 320), (256, 512)])
@pytest.mark.parametrize("stencil", [1, 2])
def test_every_size_and_block(gpu, oracle, cu, small, big, stencil):
    cfg, sf = cu
    src = _box(8, 3.615, 0.08, 3)
    reps = [_cut(src, n) for n in (1, 2, 15, 16, 17, 31, 33, 255, 257, 511, 512, 513, 1023, 1025, 2047, 2048)]
    reps += [_box(2, 3.0, 0.05, 4), _box(2, 3.615, 0.05, 5)]  # one and a few cells per edge
    tab = oracle.EamOracleTables.from_setfl(sf, 1.0, 1.0, rcut=5.0)
    F, E = _forward(oracle, reps, tab)
    with gpu.Batch(0) as b:
        b.set_eam_alloy(sf, 5.0)
        b.upload(reps)
        b.set_launch(big or 512, stencil)
        if small:
            b.set_small_block(small)
        b.run()
        d = b.download()
    assert np.sqrt(((d["F"] - F) ** 2).sum() / (F ** 2).sum()) < 1e-5
    assert np.abs(d["ep"] - E).max() < 1e-6 * np.abs(E).max()


def test_overflowing_list_and_its_gradient(gpu, oracle, cu):
    """About 300 pairs an atom where the list of a 2,048-atom replica holds
    2 x 128: forces, energies and gradient come from the cells."""
    cfg, sf = cu
    confs = [_box(8, 1.9, 0.02, 7), _box(4, 3.615, 0.08, 8)]
    rng = np.random.default_rng(5)
    pert = {k: v * rng.uniform(0.95, 1.05) for k, v in cfg["params"].items()}
    tab = oracle.EamOracleTables.from_setfl(sf, 1.0, 1.0, rcut=5.0)
    Ft, Et = _forward(oracle, confs, oracle.EamOracleTables.from_setfl(SF.tabulate(cfg, pert), 1.0, 1.0, rcut=5.0))
    F, E = _forward(oracle, confs, tab)
    n = sum(c.n for c in confs)
    dsp = oracle.EamDerivativeSplines(cfg)
    loss, grad, o = 0.0, np.zeros(9), 0
    for c in confs:
        nl = oracle.build_neighbors(c.x.copy(), c.y.copy(), c.z.copy(), c.id, c.lo, c.hi, 5.0)
        assert c.n < 2048 or np.diff(nl.off).max() > 256
        part = oracle.eam_loss_grad(c.x, c.y, c.z, nl, c.L, tab, 5.0, dsp, Ft[o:o + c.n], Et[o:o + c.n], 1.0 / n, 0.1 / n)
        loss += part[0]
        grad += part[1]
        o += c.n
    with gpu.Batch(0) as b:
        b.set_eam_alloy(sf, 5.0)
        b.set_param_derivatives(*SF.table_param_jacobian(cfg))
        b.upload(confs)
        b.set_targets(Ft, Et, 1.0 / n, 0.1 / n)
        b.run(adjoint=True)
        d = b.download()
    # pair forces of 10 to 100 eV/A that cancel to about 1: 24 bits of their sum
    scale = 300 * 100 * 2.0 ** -24
    assert np.abs(d["F"] - F).max() < 10 * scale
    assert np.abs(d["ep"] - E).max() < 2e-6 * np.abs(E).max()
    assert abs(d["loss"] - loss) < 1e-3 * loss
    assert (np.abs(d["grad"] - grad) < 1e-3 * np.abs(grad).max()).all()


@pytest.mark.parametrize("shake", [1e-6, 1e-4])
def test_pairs_at_the_cutoff(gpu, oracle, cu, shake):
    """An FCC crystal whose fourth shell lies at the cutoff, where the density
    and the pair function end with a step."""
    cfg, sf = cu
    reps = [_box(k, 5.0 / np.sqrt(2.0), shake, 11 + k, shift=0.4) for k in (2, 4, 6)]
    tab = oracle.EamOracleTables.from_setfl(sf, 1.0, 1.0, rcut=5.0)
    F, E = _forward(oracle, reps, tab)
    with gpu.Batch(0) as b:
        b.set_eam_alloy(sf, 5.0)
        b.upload(reps)
        b.run()
        d = b.download()
    # one pair on the wrong side moves an atom's energy by about 1e-3 eV
    assert np.abs(d["ep"] - E).max() < 1e-5
