"""Cutoff membership on a list that is kept while all atoms travel together: the
crystal whose fourth shell sits on the cutoff, 120 list radii from where its
list was built, against the FP64 oracle at the positions the library reports.
By pushes and by a run without rebuilds."""
import numpy as np
import pytest

from exastamp_gb300 import systems as S

pytestmark = pytest.mark.gpu

RC = 2.5
FAR = 120.0 * 2.8


@pytest.mark.parametrize("how", ["push", "run"])
@pytest.mark.parametrize("form,mixed", [("lj", False), ("lj", True), ("multi", False), ("multi", True), ("half", True)])
def test_membership_after_a_long_drift(gpu, oracle, how, form, mixed):
    a = RC / np.sqrt(2.0)
    pos, lo, hi = S.lattice(5, 5, 5, a, S.FCC_BASIS)
    rng = np.random.default_rng(11)
    pos = np.mod(pos + 0.3 * a + rng.normal(0.0, 1e-5, pos.shape), hi)
    x, y, z = (np.ascontiguousarray(pos[:, k]) for k in range(3))
    n, steps, dt = len(x), 400, 1e-6
    v = [np.full(n, s * FAR / (steps * dt)) for s in (1.0, -1.0, 0.5)]
    with gpu.Context(0) as ctx:
        ctx.set_box(lo, hi)
        ctx.set_species([1.0])
        ctx.upload(x, y, z, *v)
        if form == "multi":
            ctx.set_lj_multi(np.array([[1.0]]), np.array([[1.0]]), np.array([[RC]]), RC + 0.1)
        else:
            ctx.set_lj(1.0, 1.0, RC)
        ctx.set_skin(0.3)
        ctx.set_precision(mixed)
        if form == "half":
            ctx.set_newton3(True)
        ctx.build_neighbors()
        if how == "push":
            for _ in range(steps):
                ctx.push_f_v_r(dt)
            ctx.compute_forces(energy=False)
        else:
            ctx.run_nve(steps, dt, rebuild_every=0)
        assert ctx.list_builds() == 1
        d = ctx.download(("x", "y", "z", "ax", "ay", "az"))
    p = [np.ascontiguousarray(d[k]) for k in ("x", "y", "z")]
    assert abs(p[0].mean() - x.mean() - FAR) < 1e-3 * FAR
    w = [np.ascontiguousarray(np.mod(q, hi[k])) for k, q in enumerate(p)]
    nl = oracle.build_neighbors(*w, np.arange(n, dtype=np.uint64), lo, hi, RC + 0.3)
    ref = np.stack(oracle.lj_force(*w, nl, hi - lo, 1.0, 1.0, RC, virial=False)[:3], 1)
    got = np.stack([d["ax"], d["ay"], d["az"]], 1)
    # FP64: the wrap's rounding of the oracle's positions, 1e-13 times the shells'
    # summed stiffness of 41.5.  Mixed: two coordinates below 512, each off by at
    # most 2^-16, put a separation off by at most 5.3e-5: 2.2e-3.  A pair on the
    # wrong side is at least 0.0225.
    assert np.abs(got - ref).max() < (5e-3 if mixed else 1e-9)
