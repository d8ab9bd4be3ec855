"""Square root, reciprocal and table knot of the FP64 pair kernels against CUDA's
sqrt and division and the knot's formula: over the exponent range, on both sides
of the range that the FP32 seeds cover, exact squares, and knots at their edges."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def math(tmp_path_factory):
    import torch

    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    so = str(tmp_path_factory.mktemp("fp64") / "libfp64math.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "--cudart", "static", "-I", os.path.join(ROOT, "exastamp_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "fp64_math", "fp64_math.cu"),
                    "-o", so], check=True)
    fn = ctypes.CDLL(so).fp64_math
    vp = ctypes.c_void_p

    def run(x, nr=1000):
        x = torch.tensor(np.asarray(x, np.float64), device="cuda")
        out = {k: torch.empty_like(x) for k in ("r", "y", "r0", "inv", "sqrt", "rec", "p")}
        m = torch.empty(len(x), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        assert fn(len(x), vp(x.data_ptr()), nr, *[vp(out[k].data_ptr()) for k in ("r", "y", "r0", "inv", "sqrt", "rec")],
                  vp(m.data_ptr()), vp(out["p"].data_ptr())) == 0
        return {k: v.cpu().numpy() for k, v in out.items()} | {"m": m.cpu().numpy()}

    return run


def _ulps(a, b):
    return np.abs(a.view(np.int64) - b.view(np.int64)).max()


def test_root_and_inverse(math):
    rng = np.random.default_rng(1)
    x = [np.ldexp(rng.uniform(1.0, 2.0, 400_000), rng.integers(-95, 97, 400_000)),  # the seeds' range
         np.ldexp(rng.uniform(1.0, 2.0, 100_000), rng.integers(-4, 8, 100_000)),    # distances of a simulation
         np.arange(1.0, 20_001.0) ** 2, (np.arange(1.0, 20_001.0) / 1024.0) ** 2,   # exact squares
         1.0 + np.arange(-2000, 2000) * 2.0 ** -52, 4.0 + np.arange(-2000, 2000) * 2.0 ** -50]
    x = np.concatenate(x)
    o = math(x)
    # the last rounding is half a unit off, what precedes it some 2^-20 units:
    # at most one unit from the correctly rounded value
    assert _ulps(o["sqrt"], np.sqrt(x)) == 0 and _ulps(o["rec"], 1.0 / x) == 0
    assert _ulps(o["r"], o["sqrt"]) <= 1 and _ulps(o["r0"], o["sqrt"]) <= 1
    assert _ulps(o["inv"], o["rec"]) <= 1
    assert _ulps(o["y"], 1.0 / o["r"]) <= 1
    # exact squares have exact roots: the residual correction cannot miss them
    k = slice(500_000, 540_000)
    assert np.array_equal(o["r"][k], np.sqrt(x[k]))


def test_outside_the_seeds_range(math):
    edge = np.array([2.0 ** -95, 2.0 ** 97])
    near = np.concatenate([np.nextafter(edge, 0.0), edge, np.nextafter(edge, np.inf), edge * 0.5, edge * 2.0])
    o = math(near)
    assert _ulps(o["r"], np.sqrt(near)) <= 1 and _ulps(o["r0"], np.sqrt(near)) <= 1
    assert _ulps(o["inv"], 1.0 / near) <= 1 and _ulps(o["y"], 1.0 / np.sqrt(near)) <= 1
    far = np.array([2.0 ** -1074, 2.0 ** -1022, 1e-300, 2.0 ** -96, 2.0 ** 98, 1e300, 1.7e308, 0.0, np.inf, np.nan, -1.0])
    o = math(far)
    with np.errstate(all="ignore"):
        for k, ref in (("r", np.sqrt(far)), ("r0", np.sqrt(far)), ("inv", 1.0 / far), ("y", 1.0 / np.sqrt(far))):
            assert np.array_equal(o[k], ref, equal_nan=True), k


@pytest.mark.parametrize("nr", [5, 1000, 10_000])
def test_knot(math, nr):
    rng = np.random.default_rng(2)
    whole = np.concatenate([np.arange(1.0, min(nr, 2000) + 3.0), nr + np.arange(-3.0, 4.0), 2.0 ** np.arange(1, 31)])
    t = np.concatenate([whole, np.nextafter(whole, 0.0), np.nextafter(whole, np.inf), rng.uniform(1.0, 1.2 * nr, 50_000)])
    t = t[t >= 1.0]
    o = math(t, nr)
    m = np.minimum(np.floor(t), nr - 1)
    assert np.array_equal(o["m"], m.astype(np.int32))
    assert np.array_equal(o["p"], np.minimum(t - m, 1.0))
