"""A new density on a context that has solved or stepped already: the coarse
level's direct solve is built anew, and the graphs captured before are not
replayed on the old one's buffer.  Results equal those of a context that had
the density from the start, bit for bit."""
import numpy as np
import pytest
import torch

from anelastic_solve_b200 import abi, shear
from anelastic_solve_b200 import grid as G
from anelastic_solve_b200.mg import MGSolver
from anelastic_solve_b200.ns import NSSolver

from .helpers import compatible, field
from .test_failed_calls import zline
from .test_mg_batch import to_dev

pytestmark = pytest.mark.gpu

N = (32, 16, 64)


def density(g):
    r = np.zeros(g.ghosted, order="F")
    r[...] = np.exp(-0.05 * g.z.xc)[None, None, :]
    return r


@pytest.mark.parametrize("graph_solve", ["1", "0"])
@pytest.mark.parametrize("tol", [1e-9, 1e-11])
def test_solves(tol, graph_solve, monkeypatch):
    """Single solves and batches, the defect correction as a graph or driven
    by the host (with a captured cycle), by V-cycles and directly."""
    monkeypatch.setenv("ANEL_GRAPH_SOLVE", graph_solve)
    g = G.shear_layer_grid(*N, stretched=True)
    rhs = to_dev(compatible(field(g, np.random.default_rng(1)), g, abi.MODE_METRIC))
    p = zline(g, tol)
    p.maxcy = 8
    st = torch.cuda.Stream()

    def solves(s):
        out = []
        with torch.cuda.stream(st):
            for _ in range(3):
                out.append(torch.zeros_like(rhs))
                s.solve(out[-1], rhs, stream=st.cuda_stream)
            both = [torch.zeros_like(rhs) for _ in range(2)]
            s.solve_batch(both, [rhs, rhs], stream=st.cuda_stream)
        st.synchronize()
        return out + both

    torch.cuda.synchronize()
    used, fresh = MGSolver(g, p), MGSolver(g, p)
    solves(used)
    for s in (used, fresh):
        s.set_density(density(g))
    for a, b in zip(solves(used), solves(fresh)):
        assert torch.equal(a, b)
    used.close()
    fresh.close()


def test_steps():
    g = G.shear_layer_grid(*N, stretched=True)
    f = shear.shear_layer_fields(g, amp=1e-2)
    f["r"] = f["densityBG"] = density(g)
    names = ("u", "v", "w", "p", "rho", "scal1", "r", "densityBG")
    ns = abi.make_ns_params(Re=1000.0, Pr=1.0, g=-0.1, cfl=0.5, dtmax=1e9, ew=1, scal1_on=0)
    used, fresh = (NSSolver(g, zline(g, 1e-10), ns) for _ in range(2))
    used.set_fields({k: shear.shear_layer_fields(g, amp=1e-2)[k] for k in names})
    used.step(2)
    out = []
    for s in (used, fresh):
        s.set_clock(0.0, 0)
        s.set_fields({k: f[k] for k in names})
        s.step(2)
        out.append(s.get_fields())
        s.close()
    for k, v in out[0].items():
        np.testing.assert_array_equal(v, out[1][k], err_msg=k)
