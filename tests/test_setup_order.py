"""Contexts made, and their buffers grown, while another thread keeps the
legacy default stream busy: the clears and table uploads of a set-up are made
there, and the solves and steps that follow on the contexts' non-blocking
streams find them done."""
import threading

import pytest

from anelastic_solve_b200 import abi, shear
from anelastic_solve_b200 import grid as G
from anelastic_solve_b200.mg import MGSolver
from anelastic_solve_b200.ns import NSSolver

from .test_failed_calls import zline

pytestmark = pytest.mark.gpu


class BusyDefaultStream:
    def __enter__(self):
        self.stop = threading.Event()
        self.thread = threading.Thread(target=self.work)
        self.thread.start()

    def work(self):
        import torch

        a = torch.randn(2048, 2048, device="cuda")
        while not self.stop.is_set():
            for _ in range(20):
                a = torch.tanh(a @ a)
            torch.cuda.default_stream().synchronize()

    def __exit__(self, *exc):
        self.stop.set()
        self.thread.join()


def solves(g, rhs):
    """One solve, then batches of two and five, on a new context."""
    import torch

    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        s = MGSolver(g, zline(g, 1e-11))
        phi = [torch.zeros_like(rhs) for _ in range(8)]
        s.solve(phi[0], rhs, stream=st.cuda_stream)
        reps = [s.last_report]
        for lo, hi in ((1, 3), (3, 8)):
            reps += s.solve_batch(phi[lo:hi], [rhs] * (hi - lo), stream=st.cuda_stream)
        s.close()
    assert all(r.status == abi.OK and r.iter == 1 for r in reps)
    return phi


def steps(g, f):
    s = NSSolver(g, zline(g, 1e-11), abi.make_ns_params(Re=1000.0, Pr=1.0, g=-0.1, cfl=0.5, dtmax=1e9, ew=1))
    s.set_fields({k: f[k] for k in ("u", "v", "w", "p", "rho", "scal1", "r", "densityBG")})
    reps = [s.step(1) for _ in range(2)]
    out = [(r.dt, r.avg_div, r.max_div) for r in reps]
    s.close()
    return out


def test_set_up_beside_a_busy_default_stream():
    import torch

    g = G.shear_layer_grid(64, 32, 64, stretched=True)
    gen = torch.Generator("cuda").manual_seed(1)
    rhs = torch.zeros(g.ghosted[::-1], dtype=torch.float64, device="cuda")
    r = torch.randn(g.shape[::-1], generator=gen, dtype=torch.float64, device="cuda")
    dz = torch.from_numpy(g.z.dxc[1:-1].copy()).cuda()
    rhs[1:-1, 1:-1, 1:-1] = r - (r.mean(dim=(1, 2)) * dz).sum() / dz.sum()
    f = shear.shear_layer_fields(g, amp=1e-2)
    torch.cuda.synchronize()
    want, clock = solves(g, rhs), steps(g, f)
    torch.cuda.synchronize()
    with BusyDefaultStream():
        for _ in range(4):
            got = solves(g, rhs)
            torch.cuda.current_stream().synchronize()
            assert all(torch.equal(p, want[0]) for p in got)
            assert steps(g, f) == clock
