"""The direct fine-level solve of the mixed-precision pressure solver
(Fourier in x and y, one tridiagonal z-system per mode, FP64) against the
oracle's fine operator.

Each case asks for a tolerance that two FP64 corrections reach with room to
spare (the residual floor is about 1e-13 on these grids) and checks the
oracle's residual of the returned pressure, not the solver's own, within
1 % of that tolerance, that the direct solve alone reached it, and that the
corrections kept the mean of the starting pressure (to the rounding of the
sums, 1e-12 of its magnitude).
"""
import numpy as np
import pytest

from anelastic_solve_b200 import abi
from anelastic_solve_b200 import grid as G
from anelastic_solve_b200.mg import MGSolver
from oracle.pyoracle import OracleMG

from .helpers import compatible, field, levels_for, mg_params

pytestmark = pytest.mark.gpu

TOL = 1e-11


def to_dev(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a.T)).cuda()


def to_host(t):
    return np.asfortranarray(t.cpu().numpy().T)


def params(g, **kw):
    kw.setdefault("smoother", abi.SMOOTHER_ZLINE)
    kw.setdefault("mode", abi.MODE_METRIC)
    lv = levels_for(g)
    if kw["smoother"] == abi.SMOOTHER_ZLINE:
        lv = lv[:2] + (1,)
    return mg_params(g, levels=lv, maxcy=60, tolmax=TOL, stop=abi.STOP_RESID, **kw)


# transform lengths: one stage (4, 8), radix 2, 3, 5, the generic primes 7
# and 31, several stages; rows per z-segment 2..16, lines shorter than the
# 32 segments, a remainder, and the 64-segment form above 512
SIZES = [(4, 8, 24), (8, 4, 64), (12, 20, 33), (14, 62, 65), (96, 6, 100), (64, 32, 193), (40, 16, 257),
         (32, 8, 385), (16, 8, 512), (8, 8, 513), (256, 128, 4), (512, 4, 32)]


@pytest.mark.parametrize("n", SIZES)
def test_direct_solve_meets_the_oracles_operator(n):
    g = G.shear_layer_grid(*n, stretched=True)
    rng = np.random.default_rng(sum(n))
    src = compatible(field(g, rng), g, abi.MODE_METRIC)
    phi0 = field(g, rng)
    o = OracleMG(g, params(g))
    s = MGSolver(g, params(g, precision=abi.PREC_MIXED))
    d = to_dev(phi0)
    s.solve(d, to_dev(src))
    rep = s.last_report
    s.close()
    got = to_host(d)
    assert rep.status == abi.OK and rep.reserved == 1 and 1 <= rep.iter <= 2
    assert o.true_resid(got, src) <= 1.01 * TOL
    inner = (slice(1, -1),) * 3
    assert abs(got[inner].mean() - phi0[inner].mean()) <= 1e-12 * max(1.0, np.abs(got[inner]).max())


@pytest.mark.parametrize("case", ["dirichlet_z", "mixed_z_walls", "literal", "density"])
def test_direct_solve_boundaries_and_density(case):
    """Walls with values (not singular), the uniform-spacing operator and a
    density that falls with height (the null vector is r(z))."""
    stretched = case != "literal"
    g = G.shear_layer_grid(24, 12, 40, stretched=stretched)
    tbc, vbc = (0, 1, 0, 1, 0, 0), (0.0,) * 6
    if case == "dirichlet_z":
        tbc, vbc = (0, 2, 0, 2, 0, 0), (0.0, 0.3, 0.0, -0.2, 0.0, 0.0)
    elif case == "mixed_z_walls":
        tbc, vbc = (0, 1, 0, 2, 0, 0), (0.0, 0.4, 0.0, 0.1, 0.0, 0.0)
    mode = abi.MODE_LITERAL if case == "literal" else abi.MODE_METRIC
    kw = dict(tbc=tbc, vbc=vbc, mode=mode)
    if case == "literal":
        kw["smoother"] = abi.SMOOTHER_RBPGS
    rng = np.random.default_rng(9)
    src = compatible(field(g, rng), g, mode)
    o = OracleMG(g, params(g, **kw))
    s = MGSolver(g, params(g, precision=abi.PREC_MIXED, **kw))
    if case == "density":
        r = np.zeros(g.ghosted, order="F")
        r[...] = np.exp(-0.04 * g.z.xc)[None, None, :]
        o.set_density(r)
        s.set_density(r)
    d = to_dev(field(g, rng))
    s.solve(d, to_dev(src))
    rep = s.last_report
    s.close()
    assert rep.status == abi.OK and rep.reserved == 1
    assert o.true_resid(to_host(d), src) <= 1.01 * TOL


def test_direct_batch_equals_alone():
    """Members of a batch, one of them already solved, equal their
    one-member solves bit for bit."""
    g = G.shear_layer_grid(24, 20, 96, stretched=True)
    rng = np.random.default_rng(3)
    rhs = [to_dev(compatible(field(g, rng), g, abi.MODE_METRIC)) for _ in range(3)]
    phi0 = [to_dev(field(g, rng)) for _ in range(3)]
    s = MGSolver(g, params(g, precision=abi.PREC_MIXED))
    s.solve(phi0[1], rhs[1])
    alone, reps = [p.clone() for p in phi0], []
    for p, f in zip(alone, rhs):
        s.solve(p, f)
        reps.append(s.last_report)
    both = [p.clone() for p in phi0]
    for got, want in zip(s.solve_batch(both, rhs), reps):
        assert (got.iter, got.resid, got.status) == (want.iter, want.resid, want.status)
    s.close()
    assert reps[1].iter == 0 and reps[0].iter >= 1
    for p, q in zip(both, alone):
        np.testing.assert_array_equal(to_host(p), to_host(q))


def test_vcycles_take_over_and_stay_selectable(monkeypatch):
    """An incompatible right-hand side cannot be solved: the direct solve
    hands over to V-cycles, which report as before.  ANEL_SPECTRAL=0 keeps
    V-cycles from the start, and they are the default at 1e-10."""
    g = G.shear_layer_grid(16, 8, 64, stretched=True)
    rng = np.random.default_rng(4)
    bad = field(g, rng) + 1.0
    p = params(g, precision=abi.PREC_MIXED)
    p.maxcy = 6
    s = MGSolver(g, p)
    d = to_dev(np.zeros(g.ghosted, order="F"))
    s.solve(d, to_dev(bad))
    rep = s.last_report
    s.close()
    assert rep.status == abi.ERR_NOCONV and rep.iter == 7 and rep.reserved == 0
    src = compatible(field(g, rng), g, abi.MODE_METRIC)
    loose = params(g, precision=abi.PREC_MIXED)
    loose.tolmax = 1e-10
    for env, prm, direct in ((None, loose, 0), ("1", loose, 1), ("0", params(g, precision=abi.PREC_MIXED), 0)):
        if env is None:
            monkeypatch.delenv("ANEL_SPECTRAL", raising=False)
        else:
            monkeypatch.setenv("ANEL_SPECTRAL", env)
        s = MGSolver(g, prm)
        d = to_dev(np.zeros(g.ghosted, order="F"))
        s.solve(d, to_dev(src))
        rep = s.last_report
        s.close()
        assert rep.status == abi.OK and rep.reserved == direct and rep.resid <= prm.tolmax
