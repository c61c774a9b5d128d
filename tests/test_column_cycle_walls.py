"""The column cycle with its coarse level solved directly, under wall values
and densities that change the z-systems' null vector or leave none: as many
cycles as the FP64 cycle that relaxes down to level 1 needs, or fewer, and
the oracle's residual of the result."""
import numpy as np
import pytest

from anelastic_solve_b200 import abi
from anelastic_solve_b200 import grid as G
from anelastic_solve_b200.mg import MGSolver
from oracle.pyoracle import OracleMG

from .helpers import compatible, field, levels_for, mg_params
from .test_mg_batch import to_dev, to_host

pytestmark = pytest.mark.gpu

TOL = 1e-9


def check(n, tbc, vbc, rate):
    g = G.shear_layer_grid(*n, stretched=True)
    rng = np.random.default_rng(1)
    src = field(g, rng)
    if tbc[1] == tbc[3] == 1:
        src = compatible(src, g, abi.MODE_METRIC)
    r = np.zeros(g.ghosted, order="F")
    r[...] = np.exp(-rate * g.z.xc)[None, None, :]
    kw = dict(levels=levels_for(g)[:2] + (1,), tbc=tbc, vbc=vbc, mode=abi.MODE_METRIC,
              smoother=abi.SMOOTHER_ZLINE, maxcy=100, tolmax=TOL, stop=abi.STOP_RESID)
    iters = {}
    for prec in (abi.PREC_FP64, abi.PREC_MIXED):
        s = MGSolver(g, mg_params(g, precision=prec, **kw))
        s.set_density(r)
        phi = to_dev(np.zeros(g.ghosted, order="F"))
        s.solve(phi, to_dev(src))
        rep = s.last_report
        s.close()
        assert rep.status == abi.OK and rep.reserved == 0
        iters[prec] = rep.iter
    assert iters[abi.PREC_MIXED] <= iters[abi.PREC_FP64]
    o = OracleMG(g, mg_params(g, **kw))
    o.set_density(r)
    assert o.true_resid(to_host(phi), src) <= 1.01 * TOL


@pytest.mark.parametrize("rate", [0.0, 0.05])
@pytest.mark.parametrize("tbc", [(0, 2, 0, 2, 0, 0), (0, 1, 0, 2, 0, 0), (0, 2, 0, 1, 0, 0)])
@pytest.mark.parametrize("n", [(32, 16, 64), (64, 32, 128)])
def test_dirichlet_walls(n, tbc, rate):
    """No null vector: nothing is taken from the solution of mode (0, 0)."""
    check(n, tbc, (0, 0.2, 0, -0.1, 0, 0), rate)


@pytest.mark.parametrize("rate", [0.0, 1e-3, 0.05])
@pytest.mark.parametrize("n", [(32, 16, 64), (64, 32, 128), (16, 8, 512)])
def test_density_under_neumann_walls(n, rate):
    """The null vector is r(z) = exp(-rate z)."""
    check(n, (0, 1, 0, 1, 0, 0), (0.0,) * 6, rate)
