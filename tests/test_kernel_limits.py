"""Kernels at the largest sizes that their launches take."""
import pytest

from anelastic_solve_b200 import abi
from anelastic_solve_b200 import grid as G
from anelastic_solve_b200.mg import MGSolver

from .test_failed_calls import zline

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("members", [2047, 2048, 4100])
def test_direct_batch_of_many_members(members):
    """16x16x64 has 32 blocks of the direct solve's last pass in a column of
    blocks: 2047 members fill a launch's third dimension.  Every member
    equals its solve alone."""
    import torch

    g = G.shear_layer_grid(16, 16, 64, stretched=True)
    gen = torch.Generator("cuda").manual_seed(members)
    dz = torch.from_numpy(g.z.dxc[1:-1].copy()).cuda()
    n = 3  # right-hand sides, shared by the members; each has its own pressure
    rhs = torch.zeros((n,) + g.ghosted[::-1], dtype=torch.float64, device="cuda")
    f = torch.randn((n,) + g.shape[::-1], generator=gen, dtype=torch.float64, device="cuda")
    f -= ((f.mean(dim=(2, 3)) * dz).sum(dim=1) / dz.sum())[:, None, None, None]
    rhs[:, 1:-1, 1:-1, 1:-1] = f
    s = MGSolver(g, zline(g, 1e-11))
    want = torch.zeros_like(rhs)
    for b in range(n):
        s.solve(want[b], rhs[b])
        assert s.last_report.reserved == 1
    phi = torch.zeros((members,) + g.ghosted[::-1], dtype=torch.float64, device="cuda")
    reps = s.solve_batch(list(phi), [rhs[b % n] for b in range(members)])
    s.close()
    assert all(r.status == abi.OK and r.iter == 1 for r in reps)
    for b in range(n):
        assert torch.equal(phi[b::n], want[b].expand_as(phi[b::n]))
