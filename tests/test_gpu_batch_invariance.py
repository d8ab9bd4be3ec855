"""A replica's results do not depend on the batch it is in: the library takes other
block sizes for few and for many small replicas, and every block size must give
the same bits, from the pair list and from the cells, forward and gradient."""
import numpy as np
import pytest

from exastamp_gb300 import setfl as SF
from exastamp_gb300 import systems as S

pytestmark = pytest.mark.gpu


def _box(k, a, sig, seed, n=None):
    pos, lo, hi = S.lattice(k, k, k, a, S.FCC_BASIS)
    pos = np.mod(pos + np.random.default_rng(seed).normal(0.0, sig, pos.shape), hi)
    pos[pos >= hi] = 0.0
    pos = pos[:n]
    return S._make(pos, lo, hi, np.zeros(len(pos)), np.array([63.546]), np.zeros_like(pos), {})


def _evaluate(gpu, cfg, sf, reps, nfirst, small=0):
    """The first nfirst replicas' forward results, and loss and gradient."""
    n = sum(r.n for r in reps)
    with gpu.Batch(0) as b:
        b.set_eam_alloy(sf, 5.0)
        b.set_param_derivatives(*SF.table_param_jacobian(cfg))
        b.upload(reps)
        if small:
            b.set_small_block(small)
        rng = np.random.default_rng(1)
        b.set_targets(rng.normal(0.0, 0.5, (n, 3)), rng.normal(-3.0, 0.1, n), 0.01, 0.02)
        b.run(adjoint=True)
        d = b.download()
    m = sum(r.n for r in reps[:nfirst])
    first = [d["F"][:m], d["ep"][:m]] + [np.asarray(d[k])[:nfirst] for k in d if np.shape(d[k])[:1] == (len(reps),)]
    assert len(first) >= 4  # energies and virials of the replicas too
    return first, [np.asarray(d["loss"]), np.asarray(d["grad"])]


def test_same_bits_in_any_batch_and_block(gpu):
    cfg = SF.load_cu_params()
    sf = SF.tabulate(cfg)
    reps = [_box(6, 3.615, 0.08, n, n) for n in (1, 15, 33, 64, 65, 100, 128, 129, 243, 255, 256, 257, 400, 511, 512)]
    reps.append(_box(5, 1.7, 0.02, 9))  # 500 atoms of some 400 pairs: from the cells
    first, total = _evaluate(gpu, cfg, sf, reps, len(reps))
    for small in (64, 96, 128, 256):
        f, t = _evaluate(gpu, cfg, sf, reps, len(reps), small)
        assert all(np.array_equal(a, b) for a, b in zip(f + t, first + total)), small
    many = reps + [_box(2, 3.615, 0.08, 100 + k) for k in range(800)]
    f, _ = _evaluate(gpu, cfg, sf, many, len(reps))
    assert all(np.array_equal(a, b) for a, b in zip(f, first))
