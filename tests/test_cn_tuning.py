"""The autotuner of the Crank-Nicolson column solves."""
import pytest

from anelastic_solve_b200 import abi
from anelastic_solve_b200 import grid as G
from anelastic_solve_b200._lib import tuning_report
from anelastic_solve_b200.ns import NSSolver

from .test_failed_calls import zline

pytestmark = pytest.mark.gpu


def context(g, **kw):
    kw = {"Re": 1000.0, "Pr": 1.0, "g": -0.1, "cfl": 0.5, "dtmax": 1e9, "ew": 1, "scal1_on": 0, **kw}
    return NSSolver(g, zline(g, 1e-10), abi.make_ns_params(**kw))


def test_choices_are_kept_per_number_of_solves_in_a_launch():
    """Four variables or five with scal1; an LES launch takes four at most."""
    g = G.shear_layer_grid(24, 12, 64, stretched=True)
    for kw in (dict(), dict(scal1_on=1), dict(les=True), dict(les=True, scal1_on=1)):
        context(g, **kw).close()
    keys = [line.split(":")[0] for line in tuning_report().splitlines()]
    keys = {k.strip() for k in keys if "24x12x64" in k and k.startswith("k_cn")}
    at = "dev0 24x12x64 solves="
    assert keys == {f"k_cn_column {at}4", f"k_cn_column {at}5", f"k_cn_column_les {at}4"}


@pytest.mark.parametrize("kw", [dict(), dict(les=True, scal1_on=1)])
def test_a_tuned_context_is_a_fresh_one(kw):
    """The fields that the variants are timed on are zero again."""
    s = context(G.shear_layer_grid(40, 12, 64, stretched=True), **kw)
    names = ("u", "v", "w", "p", "rho", "scal1", "q_u", "q_v", "q_w", "q_rho", "q_s", "psrc")
    for k, v in s.get_fields(names).items():
        assert not v.any(), k
    s.close()
