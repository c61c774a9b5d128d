"""Direct solves that hand over to V-cycles: a tolerance that FP64 cannot
reach leaves every member unconverged after two corrections."""
import numpy as np
import pytest

from anelastic_solve_b200 import abi
from anelastic_solve_b200 import grid as G
from anelastic_solve_b200.mg import MGSolver

from .helpers import compatible, field
from .test_failed_calls import zline
from .test_mg_batch import to_dev

pytestmark = pytest.mark.gpu

# columns of 64 cells (column cycle, one CUDA graph) and of 40 (row-major
# cycle, driven by the host)
GRIDS = [(16, 8, 64), (16, 8, 40)]


def problem(n, maxcy, tol=1e-30):
    g = G.shear_layer_grid(*n, stretched=True)
    p = zline(g, tol)
    p.maxcy = maxcy
    return g, MGSolver(g, p), to_dev(compatible(field(g, np.random.default_rng(5)), g, abi.MODE_METRIC))


@pytest.mark.parametrize("n", GRIDS)
def test_corrections_count_towards_the_cycle_limit(n):
    """maxcy is the limit of corrections and V-cycles together: one cycle at
    3 and two at 4, seen in the launches (a cycle's are more than those of
    the hand-over's first residual)."""
    launches = {}
    for maxcy in (2, 3, 4):
        g, s, rhs = problem(n, maxcy)
        phi = rhs * 0.0
        for _ in range(2):  # the second with the graphs made
            phi.zero_()
            s.solve(phi, rhs)
        r = s.last_report
        assert r.status == abi.ERR_NOCONV and r.iter == maxcy + 1 and r.reserved == (maxcy == 2)
        launches[maxcy] = r.launches
        s.close()
    cycle = launches[4] - launches[3]
    assert cycle > 0 and launches[3] - launches[2] < 2 * cycle


def test_batch_time_holds_the_cycles():
    """ms of a batch's reports: 58 V-cycles after the two corrections, so far
    more than a quarter of a single solve's time."""
    g, s, rhs = problem(GRIDS[0], 60)
    for _ in range(2):
        s.solve(rhs * 0.0, rhs)
        alone = s.last_report.ms
        reps = s.solve_batch([rhs * 0.0 for _ in range(3)], [rhs] * 3)
    s.close()
    for r in reps:
        assert r.status == abi.ERR_NOCONV and r.ms == reps[0].ms > 0.25 * alone
