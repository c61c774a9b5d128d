"""The direct solve at its longest transforms and z-systems, and the V-cycles
that it took the place of: the mixed-precision tests again without it, where
their cycle bounds and tolerances are those of the FP32 cycles."""
import pytest

from anelastic_solve_b200 import abi
from anelastic_solve_b200.mg import MGSolver

from . import test_anelastic as anelastic
from . import test_mg_parity as mg_parity
from . import test_ns_parity as ns_parity
from . import test_spectral_solve as direct

pytestmark = pytest.mark.gpu


# z-systems of 6 rows in 32 segments, of 12 and 16 rows in 64; y transforms
# in blocks of 4 columns (above 768 points) and of 2 (above 1536), the
# longest of them; the longest x transform
@pytest.mark.parametrize("n", [(8, 8, 192), (8, 8, 768), (8, 8, 769), (8, 8, 1024), (4, 768, 8), (4, 1024, 8),
                               (4, 1536, 8), (4, 2048, 8), (2048, 4, 8)])
def test_direct_solve_at_its_largest(n):
    direct.test_direct_solve_meets_the_oracles_operator(n)


@pytest.fixture
def vcycles(monkeypatch):
    """No direct solves; the reports of the MGSolver solves that follow."""
    monkeypatch.setenv("ANEL_SPECTRAL", "0")
    reports = []
    solve = MGSolver.solve

    def recorded(self, *a, **kw):
        out = solve(self, *a, **kw)
        if self.params.precision == abi.PREC_MIXED:
            reports.append(self.last_report)
        return out

    monkeypatch.setattr(MGSolver, "solve", recorded)
    return reports


@pytest.mark.parametrize("mode", [abi.MODE_LITERAL, abi.MODE_METRIC])
def test_point_smoother(mode, vcycles):
    mg_parity.test_mixed_precision_reaches_fp64_solution(mode)
    assert vcycles and all(r.reserved == 0 and r.iter > 2 for r in vcycles)


@pytest.mark.parametrize("name", list(mg_parity.ZMIX))
def test_z_lines(name, vcycles):
    mg_parity.test_zline_mixed_precision(name)
    assert vcycles and all(r.reserved == 0 and r.iter > 2 for r in vcycles)


@pytest.mark.parametrize("case", [ns_parity.test_mixed_precision_stepper_within_tolerance,
                                  ns_parity.test_les_mixed_precision_within_tolerance,
                                  anelastic.test_ns_mixed_with_background_within_tolerance],
                         ids=lambda f: f.__name__)
def test_steppers(case, vcycles):
    case()
