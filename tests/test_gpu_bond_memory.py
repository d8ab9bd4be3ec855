"""The bond terms of one-element eam_alloy double the list's memory.  It comes back
when they are not needed any more, and forces are right without them and when
they come again."""
import numpy as np
import pytest

from exastamp_gb300 import setfl as SF
from exastamp_gb300 import systems as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leave", ["fp64", "half", "lj", "launch"])
def test_memory_of_the_bond_terms_comes_back(gpu, leave):
    import torch

    torch.cuda.init()
    sf = SF.tabulate(SF.load_cu_params())
    s = S.eam_cu_fcc(ncell=40, displace=0.05, seed=2)

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    with gpu.Context(0) as ctx:
        ctx.upload_system(s)
        ctx.set_eam_alloy(sf, 5.0, S.EV, S.EV)
        ctx.set_skin(0.3)
        ctx.set_precision(True)
        ctx.compute_forces(energy=False)
        a = ctx.download(("ax", "ay", "az"))
        held = free()
        if leave == "fp64":
            ctx.set_precision(False)
        elif leave == "half":
            ctx.set_newton3(True)  # whose accumulators take 80 bytes an atom
        elif leave == "lj":
            ctx.set_lj(0.01, 2.3, 5.0)
        else:
            ctx.set_launch(2, 128, 1)
        ctx.build_neighbors()
        # one float for each of at least 54 entries an atom
        assert free() - held > 4 * 54 * s.n - (80 * s.n if leave == "half" else 0) - (4 << 20)
        ctx.compute_forces(energy=False)
        ctx.set_precision(True)
        ctx.set_newton3(False)
        ctx.set_launch_auto()
        ctx.set_eam_alloy(sf, 5.0, S.EV, S.EV)
        ctx.compute_forces(energy=False)
        b = ctx.download(("ax", "ay", "az"))
        assert all(np.array_equal(a[k], b[k]) for k in a)
        assert abs(free() - held) < (4 << 20) + (80 * s.n if leave == "half" else 0)
