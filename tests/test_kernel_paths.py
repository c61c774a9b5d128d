"""Kernel variants and dispatch rules at the sizes where they change.

FP64 paths (the red-black cycle, the Crank-Nicolson columns, the right-hand
sides) equal the oracle bit for bit, as everywhere.  The dynamic models'
plane averages are sums in another order than the oracle's, so they agree
within 1e-9 of the largest coefficient.  A cohort's members equal the same
members stepped alone bit for bit.
"""
import numpy as np
import pytest

from anelastic_solve_b200 import abi, shear
from anelastic_solve_b200 import grid as G
from anelastic_solve_b200.mg import MGSolver
from anelastic_solve_b200.ns import NSSolver
from oracle.pyoracle import OracleMG, OracleNS

from . import test_mg_parity as mg_parity
from .helpers import compatible, field, levels_for, mg_params
from .test_ns_parity import CMP, setup_case

pytestmark = pytest.mark.gpu

NEUMANN, DIRICHLET = (0, 1, 0, 1, 0, 0), (0, 2, 0, 2, 0, 0)
# grid, levels, pre, post, walls: one plane or four per thread on the fine
# level; odd and 2-cell coarse levels; every set of coarsened directions;
# no level and several levels in the coarse block, cells of a colour up to
# its limit of 1024; levels above it with odd extents; sweep counts 0 to 3
CYCLES = [
    ((16, 8, 16), None, 2, 2, NEUMANN),
    ((32, 16, 16), None, 1, 3, DIRICHLET),
    ((128, 32, 32), None, 2, 1, NEUMANN),
    ((32, 16, 32), (2, 2, 2), 2, 2, NEUMANN),
    ((34, 18, 20), (2, 2, 2), 2, 2, NEUMANN),
    ((68, 36, 40), (3, 3, 3), 3, 0, DIRICHLET),
    ((20, 12, 96), (3, 2, 2), 2, 2, NEUMANN),
    ((4, 4, 64), (2, 2, 5), 2, 2, DIRICHLET),
    ((32, 4, 32), (5, 2, 5), 0, 2, NEUMANN),
    ((4, 32, 32), (2, 5, 5), 2, 2, NEUMANN),
    ((32, 4, 4), (5, 2, 2), 2, 2, DIRICHLET),
    ((4, 32, 4), (2, 5, 2), 2, 2, NEUMANN),
    ((32, 32, 4), (5, 5, 2), 2, 2, NEUMANN),
]


@pytest.mark.parametrize("stop", [abi.STOP_RELMAX, abi.STOP_RESID])
@pytest.mark.parametrize("n,levels,pre,post,tbc", CYCLES)
def test_fp64_cycle_shapes_bitwise(n, levels, pre, post, tbc, stop):
    g = G.shear_layer_grid(*n, stretched=True)
    kw = dict(levels=levels or levels_for(g), tbc=tbc, vbc=(0, 0.25, 0, -0.5, 0, 0), pre=pre, post=post,
              mode=abi.MODE_METRIC, maxcy=5, tolmax=1e-30, stop=stop)
    o, s = OracleMG(g, mg_params(g, **kw)), MGSolver(g, mg_params(g, **kw))
    rng = np.random.default_rng(sum(n))
    src, ref = compatible(field(g, rng), g, abi.MODE_METRIC), field(g, rng, 0.1)
    dphi, dsrc = mg_parity.to_dev(ref), mg_parity.to_dev(src)
    o.solve(ref, src.copy(order="F"))
    s.solve(dphi, dsrc)
    np.testing.assert_array_equal(mg_parity.to_host(dphi), ref)


@pytest.mark.parametrize("les", [False, True])
@pytest.mark.parametrize("n", [(40, 12, 36), (16, 8, 8), (34, 18, 20), (64, 16, 72)])
def test_narrow_column_blocks_bitwise(n, les, monkeypatch):
    """Crank-Nicolson blocks of 32 columns, and right-hand sides on tiles and
    plane counts that do not divide the grid."""
    monkeypatch.setenv("ANEL_CN_LES_VARIANT" if les else "ANEL_CN_VARIANT", "4")
    kw = dict(Re=50000.0, g=-0.1, amp=1e-2, les=True) if les else {}
    g_, o, s, f, start = setup_case(n=n, **kw)
    for _ in range(2):
        o.step()
        s.step(1)
    names = CMP + (("nuT", "kappaT", "nappaT") if les else ())
    got = s.get_fields(names)
    for name in names:
        np.testing.assert_array_equal(got[name], f[name], err_msg=name)


@pytest.mark.parametrize("case", ["filter_x_off", "filter_z_off", "periodic_temporaries"])
def test_dynamic_filter_dispatch(case):
    """A filter direction off (fused pass), and a z rule of the filtered
    temporaries that the fused pass does not take (general path)."""
    n = (34, 18, 20) if case != "periodic_temporaries" else (16, 8, 16)
    g_ = G.shear_layer_grid(*n, stretched=False)
    mgp = abi.make_mg_params(levels_for(g_), maxcy=200, tolmax=1e-10, tbc=NEUMANN, mode=abi.MODE_METRIC,
                             stop=abi.STOP_RESID)
    nsp = abi.make_ns_params(Re=50000.0, Pr=1.0, g=-0.1, dtmax=0.005, ew=1, scal1_on=1, les=True,
                             models=(abi.MODEL_DSM,) * 3, interp=abi.DIAG_LITERAL,
                             filt={"filter_x_off": (0, 1, 1), "filter_z_off": (1, 1, 0)}.get(case, (1, 1, 1)))
    if case == "periodic_temporaries":
        nsp.tb[2][0][6] = nsp.tb[2][1][6] = 3
    f = shear.shear_layer_fields(g_, amp=1e-2)
    f["scal1"][...] = 0.5 * f["rho"]
    eddy = ("nuT", "kappaT", "nappaT")
    for k in eddy:
        f[k] = np.zeros(g_.ghosted, order="F")
    o = OracleNS(g_, mgp, nsp, f)
    for name, vt in (("u", 0), ("v", 1), ("w", 2), ("rho", 4), ("scal1", 12)):
        o.ghost(f[name], vt)
    o.project()
    s = NSSolver(g_, mgp, nsp)
    s.set_fields({k: f[k] for k in ("u", "v", "w", "p", "rho", "scal1", "r", "densityBG")})
    o.step()
    s.step(1)
    got = s.get_fields(eddy)
    for k in eddy:
        ref = f[k][1:-1, 1:-1, 1:-1]
        scale = np.abs(ref).max()
        assert scale > 0, k
        np.testing.assert_allclose(got[k][1:-1, 1:-1, 1:-1], ref, rtol=1e-9, atol=1e-9 * scale, err_msg=k)


@pytest.mark.parametrize("tol", [1e-10, 1e-11])
def test_cohort_of_more_than_one_launch(tol):
    """17 members (a launch takes 16), solved by V-cycles and directly."""
    g = G.shear_layer_grid(16, 16, 64, stretched=True)
    lv = levels_for(g)
    mg = abi.make_mg_params((lv[0], lv[1], 1), maxcy=200, tolmax=tol, tbc=NEUMANN, mode=abi.MODE_METRIC,
                            stop=abi.STOP_RESID, precision=abi.PREC_MIXED, smoother=abi.SMOOTHER_ZLINE)

    def member(b):
        ns = abi.make_ns_params(Re=500.0 + 100.0 * b, Pr=1.0, g=-0.05 - 0.01 * b, cfl=0.5, dtmax=1e9, ew=1,
                                scal1_on=0)
        f = shear.shear_layer_fields(g, amp=1e-2, seed=b)
        s = NSSolver(g, mg, ns)
        s.set_fields({k: f[k] for k in ("u", "v", "w", "p", "rho", "scal1", "r", "densityBG")})
        s.project()
        return s

    names = ("u", "v", "w", "p", "rho")
    alone = []
    for b in range(17):
        s = member(b)
        rep = s.step(2)
        alone.append((s.get_fields(names), rep.dt, rep.max_div))
        s.close()
    ms = [member(b) for b in range(17)]
    reps = NSSolver.step_cohort(ms, 2)
    for b, (s, rep) in enumerate(zip(ms, reps)):
        got = s.get_fields(names)
        for k in names:
            np.testing.assert_array_equal(got[k], alone[b][0][k], err_msg=f"member {b} {k}")
        assert (rep.dt, rep.max_div) == alone[b][1:]
        s.close()


@pytest.mark.parametrize("variant", [0, 1, 2, 3, 4])
def test_vcycles_where_the_direct_solve_is_off(variant, monkeypatch):
    """The column cycle's launch variants stay reachable and converge as they
    do, with the direct solve switched off."""
    monkeypatch.setenv("ANEL_SPECTRAL", "0")
    mg_parity.test_column_sweep_variants(variant, (64, 32, 256), monkeypatch)
