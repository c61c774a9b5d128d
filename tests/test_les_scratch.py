"""The scratch of the LES column solves (a column's eliminated diagonal per
cell, for several variables at a time)."""
import numpy as np
import pytest

from anelastic_solve_b200 import abi, shear
from anelastic_solve_b200 import grid as G
from anelastic_solve_b200.ns import NSSolver

from .test_failed_calls import zline

pytestmark = pytest.mark.gpu


def les(g, scal1_on=0):
    return NSSolver(g, zline(g, 1e-11), abi.make_ns_params(Re=5e4, Pr=1.0, g=-0.1, cfl=0.5, dtmax=1e9, ew=1,
                                                           scal1_on=scal1_on, les=True))


@pytest.mark.parametrize("scal1_on", [0, 1])
def test_pressure_source_is_no_scratch(scal1_on):
    """psrc after a context's creation and after steps: what Psource wrote on
    the interior, zero on the ghosts."""
    g = G.shear_layer_grid(32, 16, 64, stretched=True)
    f = shear.shear_layer_fields(g, amp=1e-2)
    s = les(g, scal1_on)
    s.set_fields({k: f[k] for k in ("u", "v", "w", "p", "rho", "scal1", "r", "densityBG")})
    assert not s.get_fields(("psrc",))["psrc"].any()
    for _ in range(2):
        s.step(1)
        psrc = s.get_fields(("psrc",))["psrc"]
        inner = psrc[1:-1, 1:-1, 1:-1].copy()
        assert np.abs(inner).max() > 0.0
        psrc[1:-1, 1:-1, 1:-1] = 0.0
        assert not psrc.any()
    s.close()


@pytest.mark.parametrize("n", [(64, 64, 64), (256, 128, 264), (384, 192, 192), (256, 256, 256)])
def test_les_context_within_what_a_serving_job_is_charged(n):
    """Device memory of an LES context after a step, against the serving
    engine's estimate: 14 fields, 3 eddy fields, 2 of scratch, 32 bytes a cell
    for the multigrid and 64 MB."""
    import torch

    g = G.shear_layer_grid(*n, stretched=True)
    before = torch.cuda.mem_get_info()[0]
    s = les(g)
    s.step(1)
    used = before - torch.cuda.mem_get_info()[0]
    s.close()
    assert used <= np.prod(g.ghosted) * (8 * 19 + 32) + (64 << 20)
