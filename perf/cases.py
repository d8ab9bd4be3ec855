"""Performance cases of the MD hot path: what a program that uses this package
has it do, through the public entry points, from the smallest calls to the
largest.

Each case is a dict of plain values.  `listed()` gives the fixed ones, `draw()`
others of the same ranges, `prepare()` what a program holds before the call
(a context with atoms, potential and neighbour list, or a batch of replicas),
`run()` one pass, `work()` the bytes and operations that pass cannot do
without, and `exact()` the same outputs in plain FP64 torch.

Mixed-precision results (FP32 pair arithmetic) are returned in FP32, which is
what such a run's force and velocity dumps hold; FP64 runs return FP64.  Atoms
are returned in the caller's order.
"""
from __future__ import annotations

import ctypes
import json
import math
import os

import numpy as np
import torch

from exastamp_gb300 import _capi, setfl

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DA_A2_PS2 = 1.66053906660e-23                # Da A^2 / ps^2 in joules
EV = 1.602176634e-19 / DA_A2_PS2             # 1 eV in internal units
KB = 1.380649e-23 / DA_A2_PS2                # Boltzmann constant in internal units per kelvin
CU_A, CU_MASS, CU_RCUT, CU_SKIN = 3.615, 63.546, 5.0, 0.3
LJ_DENSITY, LJ_RCUT, LJ_SKIN = 0.8442, 2.5, 0.3
MIX_DENSITY = 1.2
MIX_EPS = np.array([[1.0, 1.5], [1.5, 0.5]])
MIX_SIG = np.array([[1.0, 0.8], [0.8, 0.88]])
PARAMS = ("fe", "beta", "re", "A", "B", "alpha", "kappa", "F0", "F1")


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # One force, energy and virial evaluation of a very small crystal read
        # back to the host: what a host code pays per call (latency).
        dict(name="lj_force_500", op="force", pot="lj", cells=5, cells_y=5, cells_z=5, mixed=True, virial=True,
             out="host"),
        # The 32,000-atom LJ crystal: 20 NVE steps with two list rebuilds and
        # thermo, the small simulation whose steps are launch-bound.
        dict(name="lj_nve_32k", op="nve", pot="lj", cells=20, cells_y=20, cells_z=20, mixed=True, rebuild=10),
        # A new configuration of a million atoms: list build and forces, as a
        # program does after it moved or inserted atoms.
        dict(name="lj_build_force_1m", op="build", pot="lj", cells=63, cells_y=63, cells_z=63, mixed=True,
             virial=False, out="device"),
        # Forces of the 4,000,000-atom Cu benchmark crystal, no energies: the
        # force operator of most steps.
        dict(name="eam_force_4m", op="force", pot="eam", cells=100, cells_y=100, cells_z=100, mixed=True,
             virial=False, out="device"),
        # Two-element eam_alloy in an odd-sized box, with energies and virials
        # reduced to the thermodynamic state: a thermo step.
        dict(name="alloy_thermo_ragged", op="force", pot="alloy", cells=41, cells_y=37, cells_z=59, mixed=True,
             virial=True, out="device"),
        # The headline benchmark: 20 NVE steps of the 4,000,000-atom Cu crystal.
        dict(name="eam_nve_4m", op="nve", pot="eam", cells=100, cells_y=100, cells_z=100, mixed=True, rebuild=10),
        # A middling Cu crystal with the reference's displacement-triggered
        # rebuild.
        dict(name="eam_nve_trigger_108k", op="nve", pot="eam", cells=30, cells_y=30, cells_z=30, mixed=True,
             rebuild=-1),
        # The largest workload: 16.7 million atoms of the LJ A:B mixture with
        # voids, 20 NVE steps.
        dict(name="ljmix_nve_16m", op="nve", pot="mix", cells=161, cells_y=161, cells_z=162, mixed=True, rebuild=10),
        # Plain FP64 forces, energies and virials: the accuracy reference a
        # user checks a mixed run against.
        dict(name="eam_fp64_108k", op="force", pot="eam", cells=30, cells_y=30, cells_z=30, mixed=False, virial=True,
             out="device"),
        # One step of a host code that keeps its grid in page-locked arrays:
        # state in, one NVE step, state out.
        dict(name="eam_host_step_864k", op="host", pot="eam", cells=60, cells_y=60, cells_z=60, mixed=True),
        # The parameter fit: loss and 9-parameter gradient over 256 training
        # configurations of about 243 atoms.
        dict(name="batch_grad_256", op="batch", nrep=256, nmin=236, nmax=250, adjoint=True),
        # 4,096 replicas of 32-2,048 atoms: forward and gradient.
        dict(name="batch_grad_4096", op="batch", nrep=4096, nmin=32, nmax=2048, adjoint=True),
    ]


def _cells(rng, lo, hi):
    """Unit cells per edge of a box of about lo..hi atoms (log-uniform), each
    edge drawn by itself so that boxes are ragged."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    k = (n / 4.0) ** (1.0 / 3.0)
    c = [max(4, int(round(k * rng.uniform(0.85, 1.18)))) for _ in range(3)]
    while 4 * c[0] * c[1] * c[2] > hi:
        c[c.index(max(c))] -= 1
    return dict(cells=c[0], cells_y=c[1], cells_z=c[2])


def draw(rng):
    op = rng.choice(["force", "force", "build", "nve", "nve", "host", "batch"])
    if op == "batch":
        if rng.random() < 0.4:  # a training set: equal-sized configurations
            m = rng.randint(100, 500)
            return dict(op=op, nrep=rng.randint(33, 400), nmin=m, nmax=m + 14, adjoint=rng.random() < 0.7)
        return dict(op=op, nrep=int(math.exp(rng.uniform(math.log(64), math.log(4000)))), nmin=32,
                    nmax=rng.randint(300, 2048), adjoint=rng.random() < 0.7)
    if op == "host":
        return dict(op=op, pot="eam", mixed=True, **_cells(rng, 300_000, 1_500_000))
    if op == "nve":
        pot = rng.choice(["lj", "eam", "eam", "mix"])
        return dict(op=op, pot=pot, mixed=True, rebuild=rng.choice([10, 10, -1]), **_cells(rng, 4_000, 4_000_000))
    pot = rng.choice(["lj", "eam", "eam", "alloy", "mix"])
    if op == "build":
        return dict(op=op, pot=pot, mixed=True, virial=False, out="device", **_cells(rng, 20_000, 4_000_000))
    if rng.random() < 0.3:  # small calls read back to the host
        return dict(op=op, pot=pot, mixed=True, virial=rng.random() < 0.5, out="host", **_cells(rng, 500, 9_000))
    mixed = rng.random() < 0.75
    return dict(op=op, pot=pot, mixed=mixed, virial=rng.random() < 0.4, out="device",
                **_cells(rng, 20_000, 4_000_000 if mixed else 400_000))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _dims(case):
    return int(case["cells"]), int(case["cells_y"]), int(case["cells_z"])


def _potential(case):
    """(lattice constant, masses, rcut, skin, dt, kB T, displacement) of the case's system."""
    pot = case["pot"]
    if pot == "lj":
        return (4.0 / LJ_DENSITY) ** (1.0 / 3.0), [1.0], LJ_RCUT, LJ_SKIN, 0.005, 1.0, 0.06
    if pot == "mix":
        return (4.0 / MIX_DENSITY) ** (1.0 / 3.0), [1.0, 1.0], 2.5, 0.3, 0.002, 1.0, 0.05
    masses = [CU_MASS] if pot == "eam" else [CU_MASS, 58.693]
    return CU_A, masses, CU_RCUT, CU_SKIN, 1e-3, KB * 300.0, 0.08


def _atoms(case, seed):
    """Seeded atoms on the GPU: an FCC crystal (z slowest, as a cell grid holds
    its atoms) with thermal displacements (at most 2.5 sigma, so that no two
    atoms overlap) and velocities; the mixture has 80:20 types and spherical
    voids, the alloy half and half.  Returns x (3, n), v (3, n), type (n,) or
    None, L (3,); n is the case's, whatever the seed."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(1_000_003 * int(seed) + 17)
    a, masses, _, _, _, kT, disp = _potential(case)
    nx, ny, nz = _dims(case)
    L = torch.tensor([nx * a, ny * a, nz * a], dtype=torch.float64, device=dev)
    basis = torch.tensor([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]], dtype=torch.float64, device=dev)
    k, j, i = torch.meshgrid(torch.arange(nz, device=dev), torch.arange(ny, device=dev),
                             torch.arange(nx, device=dev), indexing="ij")
    cell = torch.stack([i, j, k], 0).reshape(3, -1, 1).double()
    x = ((cell + basis.T[:, None, :] + 0.25) * a).reshape(3, -1)
    if case["pot"] == "mix":  # voids: one sphere of radius 8 per 262,144 atoms
        nv = max(1, round(x.shape[1] / 262_144))
        c = torch.as_tensor(np.random.default_rng(nv).random((nv, 3)), device=dev) * L
        r = min(8.0, 0.2 * float(L.min()))
        keep = torch.ones(x.shape[1], dtype=torch.bool, device=dev)
        for q in range(nv):
            d = x - c[q][:, None]
            d -= L[:, None] * torch.round(d / L[:, None])
            keep &= (d * d).sum(0) > r * r
        x = x[:, keep]
    x = x + disp * torch.randn(x.shape, dtype=torch.float64, device=dev, generator=g).clamp_(-2.5, 2.5)
    x = x - L[:, None] * torch.floor(x / L[:, None])
    x = torch.where(x >= L[:, None], torch.zeros_like(x), x).contiguous()
    n = x.shape[1]
    t = None
    m = torch.full((n,), masses[0], dtype=torch.float64, device=dev)
    if len(masses) > 1:
        frac = 0.2 if case["pot"] == "mix" else 0.5
        t = (torch.rand(n, device=dev, generator=g) < frac).to(torch.uint8)
        m = torch.where(t > 0, masses[1], masses[0]).double()
    v = torch.randn((3, n), dtype=torch.float64, device=dev, generator=g) * torch.sqrt(kT / m)
    v = (v - (v * m).sum(1, keepdim=True) / m.sum()).contiguous()
    return x, v, t, L


def _tables(nel, scale=None, taper=True):
    """Analytic Cu-like EAM tables (and a second, slightly different element)
    on setfl knots: the parameters of data/cu_analytic.json.  With `taper` the
    density and the pair function go smoothly to zero over the last 0.5 A, as
    those of published setfl files do; the parameter fit's are plain."""
    with open(os.path.join(ROOT, "data", "cu_analytic.json")) as fh:
        cfg = json.load(fh)
    nr, nrho, rcut, rho_e = int(cfg["nr"]), int(cfg["nrho"]), float(cfg["rcut"]), float(cfg["rho_e"])
    dr, drho = rcut / (nr - 1), float(cfg["rhomax_over_rho_e"]) * rho_e / (nrho - 1)
    r, rho = np.arange(nr) * dr, np.arange(nrho) * drho
    els = []
    for e in range(nel):
        p = dict(cfg["params"])
        if e == 1:
            p.update(fe=0.9 * p["fe"], A=1.05 * p["A"], B=0.97 * p["B"], F0=1.04 * p["F0"])
        if scale:
            p = {k: v * scale.get(k, 1.0) for k, v in p.items()}
        els.append(p)
    F = [-p["F0"] * np.sqrt(rho / rho_e) + p["F1"] * (rho / rho_e) for p in els]
    f = [p["fe"] * np.exp(-p["beta"] * (r / p["re"] - 1.0)) for p in els]
    phi = [p["A"] * np.exp(-p["alpha"] * (r / p["re"] - 1.0)) - p["B"] * np.exp(-p["kappa"] * (r / p["re"] - 1.0))
           for p in els]
    if taper:
        u = np.clip((rcut - r) / 0.5, 0.0, 1.0)
        f, phi = ([q * (u * u * u * (10.0 + u * (6.0 * u - 15.0))) for q in t] for t in (f, phi))
    z = [0.5 * r * (phi[a] + phi[b]) for a in range(nel) for b in range(a + 1)]
    return dict(nrho=nrho, drho=drho, nr=nr, dr=dr, rcut=rcut, F=F, f=f, z=z)


def _setfl(tab):
    n = len(tab["F"])
    return setfl.Setfl(["Cu", "Ni"][:n], [29, 28][:n], [CU_MASS, 58.693][:n], [CU_A, 3.52][:n], ["fcc"] * n,
                       tab["nrho"], tab["drho"], tab["nr"], tab["dr"], tab["rcut"], tab["F"], tab["f"], tab["z"])


def _replicas(case, seed):
    """Independent copper-like replicas: FCC or BCC, up to 3% strain, thermal
    displacements, log-uniform target sizes, vacancies down to the target where
    the lattice has more sites.  Lattices and sizes are the case's, strains,
    vacancies and displacements the seed's.  Returns a list of (positions (n,
    3), L (3,))."""
    size = np.random.default_rng(int(case["nrep"]))
    rng = np.random.default_rng(7919 * int(seed) + 3)
    fcc = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    bcc = np.array([[0, 0, 0], [0.5, 0.5, 0.5]])
    out = []
    for _ in range(int(case["nrep"])):
        target = int(round(math.exp(size.uniform(math.log(case["nmin"]), math.log(case["nmax"])))))
        basis, a = (fcc, CU_A) if size.random() < 0.5 else (bcc, 2.87)
        k = max(1, int(math.ceil((target / len(basis)) ** (1.0 / 3.0) - 0.3)))
        d = [k, k, max(1, int(math.ceil(target / (len(basis) * k * k) - 0.05)))]
        while min(d) * a < 5.2:
            d[d.index(min(d))] += 1
        box = np.array(d) * a * (1.0 + rng.uniform(-0.03, 0.03, 3))
        g = np.stack(np.meshgrid(*[np.arange(m) for m in d], indexing="ij"), -1).reshape(-1, 3)
        x = ((g[:, None, :] + basis[None, :, :]).reshape(-1, 3) + 0.25) / np.array(d) * box
        if len(x) > target >= 0.93 * len(x):
            x = x[np.sort(rng.permutation(len(x))[:target])]
        x = x[: int(case["nmax"]) if case["nmax"] > 1024 else 2048]
        x = x + rng.normal(0.0, rng.uniform(0.05, 0.12), x.shape)
        x = x - box * np.floor(x / box)
        x[x >= box] = 0.0
        out.append((x, box))
    return out


class _Replica:
    """What Batch.upload reads of a system."""

    def __init__(self, x, box):
        self.n = len(x)
        self.x, self.y, self.z = (np.ascontiguousarray(x[:, k]) for k in range(3))
        self.lo, self.hi = np.zeros(3), box


# parameters of the fit's targets: every one off by up to 10%
TARGET_SCALE = dict(fe=1.04, beta=0.97, re=1.01, A=1.06, B=0.95, alpha=1.03, kappa=1.02, F0=0.96, F1=1.07)

_stream = None


def _the_stream():
    """The program's one CUDA stream."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def prepare(case, seed):
    st = _the_stream()
    if case["op"] == "batch":
        reps = [_Replica(x, L) for x, L in _replicas(case, seed)]
        n = sum(r.n for r in reps)
        b = _capi.Batch(0, st.cuda_stream)
        b.upload(reps)
        if case["adjoint"]:
            b.set_eam_alloy(_setfl(_tables(1, TARGET_SCALE, taper=False)), CU_RCUT)
            b.run()
            t = b.download()
            b.set_eam_alloy(_setfl(_tables(1, taper=False)), CU_RCUT)
            b.set_param_derivatives(*setfl.table_param_jacobian(setfl.load_cu_params()))
            b.set_targets(t["F"], t["ep"], 1.0 / n, 0.1 / n)
        else:
            b.set_eam_alloy(_setfl(_tables(1, taper=False)), CU_RCUT)
        # page-locked result arrays, which such a program keeps, and the
        # single-precision copies that go into its logs
        host = [torch.empty(n, dtype=torch.float64, pin_memory=True) for _ in range(4)]
        return dict(case=case, b=b, n=n, host=host, rep=np.empty(len(reps)), vir=np.empty((len(reps), 9)),
                    grad=np.empty(9), f32=[torch.empty(n, dtype=torch.float32) for _ in range(4)])
    x, v, t, L = _atoms(case, seed)
    _, masses, rcut, skin, dt, _, _ = _potential(case)
    ctx = _capi.Context(0, st.cuda_stream)
    ctx.set_box(np.zeros(3), L.cpu().numpy())
    ctx.set_species(masses)
    xh, vh = x.cpu().numpy(), v.cpu().numpy()
    ctx.upload(*xh, *vh, types=None if t is None else t.cpu().numpy())
    if case["pot"] == "lj":
        ctx.set_lj(1.0, 1.0, rcut)
    elif case["pot"] == "mix":
        ctx.set_lj_multi(MIX_EPS, MIX_SIG, 2.5 * MIX_SIG)
    else:
        ctx.set_eam_alloy(_setfl(_tables(len(masses))), rcut, EV, EV)
    ctx.set_skin(skin)
    ctx.build_neighbors()
    s = dict(case=case, ctx=ctx, n=x.shape[1], dt=dt, seen={}, stream=st)
    if case["op"] == "host":
        ctx.set_precision(False)
        ctx.compute_forces(energy=False)
        d = ctx.download(("ax", "ay", "az"))
        s["pinned"] = {}
        for k, a in zip(("x", "y", "z", "vx", "vy", "vz"), list(xh) + list(vh)):
            s["pinned"][k] = torch.from_numpy(a).pin_memory()
        for k in ("ax", "ay", "az"):
            s["pinned"][k] = torch.from_numpy(d[k]).pin_memory()
        s["grid"] = {k: p.numpy() for k, p in s["pinned"].items()}
        s["f32"] = [torch.empty(s["n"], dtype=torch.float32) for _ in range(6)]
    ctx.set_precision(bool(case["mixed"]))
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
class _Dev:
    def __init__(self, ptr, n, kind):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (n,), "typestr": kind, "version": 3}


def _device_arrays(s, names):
    """The context's device arrays (zero copy) and the caller index of each row."""
    ctx = s["ctx"]
    p = [ctypes.c_void_p() for _ in range(11)]
    ctx._chk(ctx._L.gbmd_device_state(ctx.h, *[ctypes.byref(q) for q in p]))
    keys = ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az", "ep")

    def view(ptr, kind):
        if (ptr, kind) not in s["seen"]:  # two buffers each, at most
            s["seen"][ptr, kind] = torch.as_tensor(_Dev(ptr, s["n"], kind), device="cuda")
        return s["seen"][ptr, kind]

    return [view(p[keys.index(k)].value, "<f8") for k in names], view(p[10].value, "<i4")


def _in_caller_order(s, names, dtype):
    rows, user = _device_arrays(s, names)
    out = torch.empty((len(rows), s["n"]), dtype=dtype, device="cuda")
    return out.index_copy_(1, user.long(), torch.stack(rows).to(dtype))


def run(s):
    case = s["case"]
    if case["op"] == "batch":
        b = s["b"]
        b.run(adjoint=bool(case["adjoint"]), use_graph=True)
        loss = ctypes.c_double()
        b._chk(b._L.gbmd_batch_download(b.h, *[h.data_ptr() for h in s["host"]], s["rep"].ctypes.data,
                                        s["vir"].ctypes.data, ctypes.addressof(loss), s["grad"].ctypes.data))
        for h, f in zip(s["host"], s["f32"]):
            f.copy_(h)
        out = dict(f=list(s["f32"]), e=s["rep"].astype(np.float32), vir=s["vir"].astype(np.float32))
        if case["adjoint"]:
            out.update(loss=np.float32(loss.value), grad=s["grad"].astype(np.float32))
        return out
    ctx = s["ctx"]
    if case["op"] == "host":
        ctx.run_nve_host(s["grid"], 1, s["dt"], 10)
        for k, f in zip(("vx", "vy", "vz", "ax", "ay", "az"), s["f32"]):
            f.copy_(s["pinned"][k])
        return dict(r=[s["grid"][k] for k in ("x", "y", "z")], va=list(s["f32"]))
    dtype = torch.float32 if case["mixed"] else torch.float64
    with torch.cuda.stream(s["stream"]):
        if case["op"] == "nve":
            rows = ctx.run_nve(20, s["dt"], int(case["rebuild"]), 20, use_graph=True)
            state = _in_caller_order(s, ("x", "y", "z", "vx", "vy", "vz"), dtype)
            return dict(r=state[:3], v=state[3:], thermo=rows.astype(np.float32))
        if case["op"] == "build":
            ctx.build_neighbors()
        virial = bool(case["virial"])
        ctx.compute_forces(energy=virial, virial=virial)
        names = ("ax", "ay", "az", "ep") if virial else ("ax", "ay", "az")
        if case["out"] == "host":
            d = ctx.download(names, virial=virial)
            return {k: a.astype(np.float32 if case["mixed"] else np.float64) for k, a in d.items()}
        state = _in_caller_order(s, names, dtype)
        out = dict(a=state[:3])
        if virial:
            out.update(ep=state[3], thermo=ctx.thermo().astype(np.float32 if case["mixed"] else np.float64))
        return out


# ---------------------------------------------------------------------------
# the work of one pass
# ---------------------------------------------------------------------------
def work(case):
    if case["op"] == "batch":
        lo, hi = float(case["nmin"]), float(case["nmax"])
        n = case["nrep"] * ((hi - lo) / math.log(hi / lo))
        pairs = 21.0 * n  # unordered pairs inside the cutoff
        io = n * (24 + 32 + (32 if case["adjoint"] else 0))
        return dict(bytes=io, flops=pairs * (74 + (120 if case["adjoint"] else 0)))
    nx, ny, nz = _dims(case)
    n = 4.0 * nx * ny * nz
    a, _, rcut, skin, _, _, _ = _potential(case)
    density = 4.0 / a ** 3
    entries = density * 4.18879 * (rcut + skin) ** 3   # list entries per atom
    pairs = density * 4.18879 * rcut ** 3 / 2          # unordered pairs inside the cutoff
    flops = (35.0 if case["pot"] in ("lj", "mix") else 74.0) * pairs + 14.0
    force = 4 * entries + 24 + 24 + (80 if case.get("virial") else 0)
    if case["op"] == "host":
        return dict(bytes=n * (4 * entries + 144), flops=n * flops)
    if case["op"] == "nve":
        return dict(bytes=n * (20 * (4 * entries + 144) + 2 * 4 * entries), flops=n * 20 * flops)
    build = 4 * entries + 24 if case["op"] == "build" else 0
    return dict(bytes=n * (force + build), flops=n * flops)


# ---------------------------------------------------------------------------
# the same in plain FP64 torch
# ---------------------------------------------------------------------------
def _pairs(x, L, R):
    """Ordered pairs (i, j, image code) within R of each other as chunks of
    int32, int32, int8; the image of j is LUT[code], see _shifts."""
    dev, n = x.device, x.shape[1]
    Lh = L.tolist()
    nc = [max(1, int(l / (R * 1.0000001))) for l in Lh]
    c = [(x[d] * (nc[d] / Lh[d])).long().clamp_(0, nc[d] - 1) for d in range(3)]
    lin = (c[2] * nc[1] + c[1]) * nc[0] + c[0]
    order = torch.argsort(lin)
    lin = lin[order]
    ncell = nc[0] * nc[1] * nc[2]
    count = torch.bincount(lin, minlength=ncell)
    start = torch.cumsum(count, 0) - count
    m = int(count.max())
    table = torch.full((ncell, m), -1, dtype=torch.int64, device=dev)
    table[lin, torch.arange(n, device=dev) - start[lin]] = order
    out, step = [], max(1, 40_000_000 // (m * m))
    far = torch.tensor(1e9, dtype=torch.float64, device=dev)
    for b in range(0, ncell, step):
        cell = torch.arange(b, min(b + step, ncell), device=dev)
        cx, cy, cz = cell % nc[0], (cell // nc[0]) % nc[1], cell // (nc[0] * nc[1])
        home = table[cell]
        ph = [torch.where(home >= 0, x[d][home.clamp(min=0)], far) for d in range(3)]
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    im, nb = [], 0
                    for q, d, s in ((cz, dz, 2), (cy, dy, 1), (cx, dx, 0)):
                        w = torch.div(q + d, nc[s], rounding_mode="floor")
                        im.insert(0, w)
                        nb = nb * nc[s] + (q + d - w * nc[s])
                    other = table[nb]
                    d2 = 0
                    for s in range(3):
                        po = torch.where(other >= 0, x[s][other.clamp(min=0)] + im[s][:, None] * Lh[s], -far)
                        e = po[:, None, :] - ph[s][:, :, None]
                        d2 = d2 + e * e
                    mask = d2 <= R * R
                    if dx == dy == dz == 0:
                        mask &= ~torch.eye(m, dtype=torch.bool, device=dev)
                    h, i, j = mask.nonzero(as_tuple=True)
                    if len(h):
                        code = ((im[2] + 1) * 3 + im[1] + 1) * 3 + im[0] + 1
                        out.append((home[h, i].int(), other[h, j].int(), code[h].to(torch.int8)))
    merged, part, size = [], [], 0
    for p in out + [None]:
        if p is not None:
            part.append(p)
            size += len(p[0])
        if part and (p is None or size > 30_000_000):
            merged.append(tuple(torch.cat(q) for q in zip(*part)))
            part, size = [], 0
    return merged


def _shifts(L):
    k = torch.arange(27, device=L.device)
    return torch.stack([k % 3 - 1, (k // 3) % 3 - 1, k // 9 - 1]).double() * L[:, None]


def _spline(values, delta):
    """The setfl spline (LAMMPS array2spline) of a table: rows c3, c4, c5, c6 per
    knot 0..n (knot 0 unused), value ((c3 p + c4) p + c5) p + c6."""
    n = values.shape[0]
    f = torch.cat([values.new_zeros(1), values])
    s = torch.zeros_like(f)
    z = [f[2] - f[1], 0.5 * (f[3] - f[1])]
    mid = ((f[1:n - 3] - f[5:n + 1]) + 8.0 * (f[4:n] - f[2:n - 2])) / 12.0
    s = torch.cat([f.new_zeros(1), torch.stack(z), mid, torch.stack([0.5 * (f[n] - f[n - 2]), f[n] - f[n - 1]])])
    d = f[2:] - f[1:-1]
    c4 = 3.0 * d - 2.0 * s[1:-1] - s[2:]
    c3 = s[1:-1] + s[2:] - 2.0 * d
    pad = f.new_zeros(1)
    return torch.stack([torch.cat([pad, c3, pad]), torch.cat([pad, c4, pad]), s, f], 1)


def _lookup(r, delta, nknot, low=0):
    t = r / delta + 1.0
    m = t.long().clamp(low, nknot - 1)
    return m, (t - m).clamp(max=1.0)


def _value(c, p):
    return ((c[..., 0] * p + c[..., 1]) * p + c[..., 2]) * p + c[..., 3]


def _slope(c, p, delta):
    return ((3.0 * c[..., 0] * p + 2.0 * c[..., 1]) * p + c[..., 2]) / delta


class _Eam:
    def __init__(self, tab, dev):
        t = lambda a: torch.as_tensor(np.stack(a), dtype=torch.float64, device=dev)  # noqa: E731
        self.nel, self.nr, self.nrho, self.dr, self.drho = len(tab["F"]), tab["nr"], tab["nrho"], tab["dr"], tab["drho"]
        self.F = torch.stack([_spline(q, self.drho) for q in t(tab["F"])])
        self.f = torch.stack([_spline(q, self.dr) for q in t(tab["f"])])
        self.z = torch.stack([_spline(q, self.dr) for q in t(tab["z"])])

    def embed(self, rho, t):
        m, p = _lookup(rho, self.drho, self.nrho, 1)
        c = self.F[t, m]
        top = (self.nrho - 1) * self.drho
        dF = _slope(c, p, self.drho)
        return _value(c, p) + torch.where(rho > top, dF * (rho - top), torch.zeros_like(rho)), dF

    def zpair(self, a, b):
        hi, lo = torch.maximum(a, b), torch.minimum(a, b)
        return hi * (hi + 1) // 2 + lo


def _forces(case, x, t, L, chunks):
    """(f (3, n), energy (n,), virial (9,)) of the case's potential; the virial
    is per atom (n, 9) for results read back to the host."""
    n, dev = x.shape[1], x.device
    lut, pot = _shifts(L), case["pot"]
    t = torch.zeros(n, dtype=torch.int64, device=dev) if t is None else t.long()
    f = torch.zeros((n, 3), dtype=torch.float64, device=dev)
    e = torch.zeros(n, dtype=torch.float64, device=dev)
    per_atom = case.get("out") == "host"
    vir = torch.zeros((n, 9) if per_atom else (3, 3), dtype=torch.float64, device=dev)
    rcut = _potential(case)[2]

    def inside():
        for i, j, code in chunks:
            i, j, code = i.long(), j.long(), code.long()
            d = torch.stack([(x[s][j] + lut[s][code]) - x[s][i] for s in range(3)], 1)
            r2 = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
            k = r2 <= rcut * rcut
            yield i[k], j[k], d[k], torch.sqrt(r2[k])

    def add(i, d, scale, phi):
        nonlocal vir
        fe = d * scale[:, None]
        f.index_add_(0, i, fe)
        e.index_add_(0, i, 0.5 * phi)
        if per_atom:
            vir.index_add_(0, i, (-0.5 * fe[:, :, None] * d[:, None, :]).reshape(-1, 9))
        else:
            vir -= 0.5 * fe.T @ d

    if pot in ("lj", "mix"):
        tab = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
        eps, sig = (tab(MIX_EPS), tab(MIX_SIG)) if pot == "mix" else (tab([[1.0]]), tab([[1.0]]))
        rc = 2.5 * sig if pot == "mix" else tab([[rcut]])
        for i, j, d, r in inside():
            a, b = t[i], t[j]
            k = r <= rc[a, b]
            i, d, r, ee, s, rr = i[k], d[k], r[k], eps[a, b][k], sig[a, b][k], rc[a, b][k]
            s6, c6 = (s / r) ** 6, (s / rr) ** 6
            add(i, d, -24.0 * ee * (2.0 * s6 * s6 - s6) / (r * r), 4.0 * ee * ((s6 * s6 - s6) - (c6 * c6 - c6)))
        return f.T, e, vir.reshape(-1, 9).squeeze(0)
    E = _Eam(_tables(1 if pot == "eam" else 2), dev)
    rho = torch.zeros(n, dtype=torch.float64, device=dev)
    for i, j, d, r in inside():
        m, p = _lookup(r, E.dr, E.nr)
        rho.index_add_(0, i, _value(E.f[t[j], m], p))
    emb, dF = E.embed(rho, t)
    for i, j, d, r in inside():
        m, p = _lookup(r, E.dr, E.nr)
        c = E.z[E.zpair(t[i], t[j]), m]
        phi = _value(c, p) / r
        psi = dF[i] * _slope(E.f[t[j], m], p, E.dr) + dF[j] * _slope(E.f[t[i], m], p, E.dr) \
            + (_slope(c, p, E.dr) - phi) / r
        add(i, d, EV * psi / r, EV * phi)
    return f.T, e + EV * emb, vir.reshape(-1, 9).squeeze(0)


def _thermo(x, v, m, e, vir):
    ke = 0.5 * (v * m) @ v.T
    return torch.cat([vir, ke.reshape(9), (v * m).sum(1), torch.diagonal(ke), e.sum()[None], m.sum()[None],
                      m.new_tensor([float(len(m))])])


def _exact_batch(case, seed):
    """Forces, energies, virials, loss and parameter gradient of the replicas;
    the gradient by differentiating through tables, splines and forces."""
    dev = torch.device("cuda")
    reps = _replicas(case, seed)
    n = sum(len(x) for x, _ in reps)
    with open(os.path.join(ROOT, "data", "cu_analytic.json")) as fh:
        cfg = json.load(fh)
    tab = _tables(1, taper=False)
    r = torch.arange(tab["nr"], dtype=torch.float64, device=dev) * tab["dr"]
    rho = torch.arange(tab["nrho"], dtype=torch.float64, device=dev) * tab["drho"]
    rho_e = float(cfg["rho_e"])

    def model(theta):
        q = dict(zip(PARAMS, theta))
        u = r / q["re"] - 1.0
        E = _Eam(tab, dev)
        E.F = _spline(-q["F0"] * torch.sqrt(rho / rho_e) + q["F1"] * (rho / rho_e), E.drho)[None]
        E.f = _spline(q["fe"] * torch.exp(-q["beta"] * u), E.dr)[None]
        E.z = _spline(r * (q["A"] * torch.exp(-q["alpha"] * u) - q["B"] * torch.exp(-q["kappa"] * u)), E.dr)[None]
        return E

    def evaluate(E, m, i, j, d, rr):
        k, p = _lookup(rr, E.dr, E.nr)
        zero = torch.zeros(m, dtype=torch.float64, device=dev)
        cf, cz = E.f[0][k], E.z[0][k]
        emb, dF = E.embed(zero.index_add(0, i, _value(cf, p)), 0)
        phi = _value(cz, p) / rr
        psi = (dF[i] + dF[j]) * _slope(cf, p, E.dr) + (_slope(cz, p, E.dr) - phi) / rr
        fe = d * (psi / rr)[:, None]
        return zero[:, None].repeat(1, 3).index_add(0, i, fe), emb + zero.index_add(0, i, 0.5 * phi), fe

    theta = torch.tensor([cfg["params"][k] for k in PARAMS], dtype=torch.float64, device=dev, requires_grad=True)
    aim = model([cfg["params"][k] * TARGET_SCALE[k] for k in PARAMS])
    F, EP, erep, vrep, loss, grad = [], [], [], [], 0.0, torch.zeros(9, dtype=torch.float64, device=dev)
    group, size = [], 0
    for q, (x, L) in enumerate(reps + [(None, None)]):
        if x is not None:
            group.append((x, L))
            size += len(x)
        if not group or (x is not None and size < 60_000):
            continue
        ii, jj, dd, which, base = [], [], [], [], 0
        for w, (xr, Lr) in enumerate(group):
            X = torch.as_tensor(xr, device=dev)
            span = [(0,) if l >= 2.0 * CU_RCUT else (-1, 0, 1) for l in Lr]
            d = X[None, :, :] - X[:, None, :]
            Lt = torch.as_tensor(Lr, device=dev)
            for s in range(3):
                if len(span[s]) == 1:
                    d[..., s] -= Lt[s] * torch.round(d[..., s] / Lt[s])
            for a in span[0]:
                for b in span[1]:
                    for c in span[2]:
                        e = d + Lt * torch.tensor([a, b, c], dtype=torch.float64, device=dev)
                        r2 = (e * e).sum(2)
                        i, j = ((r2 <= CU_RCUT ** 2) & (r2 > 0)).nonzero(as_tuple=True)
                        ii.append(i + base)
                        jj.append(j + base)
                        dd.append(e[i, j])
            which += [w] * len(xr)
            base += len(xr)
        i, j, d = torch.cat(ii), torch.cat(jj), torch.cat(dd)
        rr, which = d.norm(dim=1), torch.tensor(which, device=dev)
        with torch.set_grad_enabled(bool(case["adjoint"])):
            f, ep, fe = evaluate(model(theta.unbind()), base, i, j, d, rr)
            if case["adjoint"]:
                with torch.no_grad():
                    ft, et, _ = evaluate(aim, base, i, j, d, rr)
                part = ((f - ft) ** 2).sum() / n + 0.1 * ((ep - et) ** 2).sum() / n
                grad += torch.autograd.grad(part, theta)[0]
                loss += float(part.detach())
        F.append(f.detach())
        EP.append(ep.detach())
        zero = torch.zeros(len(group), dtype=torch.float64, device=dev)
        erep.append(zero.index_add(0, which, ep.detach()))
        pair = (-0.5 * fe.detach()[:, :, None] * d[:, None, :]).reshape(-1, 9)
        vrep.append(zero[:, None].repeat(1, 9).index_add(0, which[i], pair))
        group, size = [], 0
    F = torch.cat(F)
    out = dict(f=[F[:, 0], F[:, 1], F[:, 2], torch.cat(EP)], e=torch.cat(erep), vir=torch.cat(vrep))
    if case["adjoint"]:
        out.update(loss=np.float64(loss), grad=grad)
    return out


def exact(case, seed):
    if case["op"] == "batch":
        return _exact_batch(case, seed)
    x, v, t, L = _atoms(case, seed)
    _, masses, rcut, skin, dt, kT, _ = _potential(case)
    m = torch.as_tensor(masses, dtype=torch.float64, device=x.device)[0 if t is None else t.long()].expand(x.shape[1])
    if case["op"] in ("force", "build"):
        f, e, vir = _forces(case, x, t, L, _pairs(x, L, rcut))
        out = dict(a=f / m)
        if case["virial"]:
            out.update(ep=e, thermo=_thermo(x, v, m, e, vir if case["out"] != "host" else vir.sum(0)))
        if case["out"] == "host":
            out = {k: (f / m)[s] for s, k in enumerate(("ax", "ay", "az"))}
            if case["virial"]:
                out.update(ep=e, vir=vir)
        return out
    steps = 20 if case["op"] == "nve" else 1
    # a margin for what two atoms can approach each other by in the steps
    fast = 6.0 * math.sqrt(kT / min(masses)) * dt * steps
    chunks = _pairs(x, L, rcut + 2.0 * fast)
    f, e, vir = _forces(case, x, t, L, chunks)
    rows, a = [_thermo(x, v, m, e, vir)], f / m
    box, ref, wrap = L[:, None], x.clone(), torch.zeros_like(x)
    every = int(case.get("rebuild", 0))
    for k in range(1, steps + 1):
        x = x + v * dt + a * (0.5 * dt * dt)
        v = v + a * (0.5 * dt)
        moved = every < 0 and bool((((x + wrap - ref) ** 2).sum(0) > (0.5 * skin) ** 2).any())
        if moved or (every > 0 and k % every == 0):
            # a list rebuild brings the atoms that left the box back into it
            now = x + wrap
            wrap = wrap + torch.where(now < 0, box, torch.zeros_like(x)) - torch.where(now >= box, box, torch.zeros_like(x))
            ref = x + wrap
        f, e, vir = _forces(case, x, t, L, chunks)
        a = f / m
        v = v + a * (0.5 * dt)
    r = x + wrap
    if case["op"] == "host":
        return dict(r=[r[0], r[1], r[2]], va=[v[0], v[1], v[2], a[0], a[1], a[2]])
    rows.append(_thermo(x, v, m, e, vir))
    return dict(r=r, v=v, thermo=torch.stack(rows))
