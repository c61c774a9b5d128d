"""Direct solves that hand over to V-cycles: a tolerance that FP64 cannot
reach leaves every member unconverged after two corrections."""
import numpy as np
import pytest
import torch

from anelastic_solve_b200 import abi
from anelastic_solve_b200 import grid as G
from anelastic_solve_b200._lib import lib
from anelastic_solve_b200.mg import MGSolver

from .helpers import compatible, field
from .test_failed_calls import memory_left, zline
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


def members(g):
    """Right-hand sides of a batch: incompatible (the first, third and last),
    solvable, not finite."""
    rng = np.random.default_rng(7)
    good = compatible(field(g, rng), g, abi.MODE_METRIC)
    bad = [np.asfortranarray(good + 0.1 * field(g, rng) + q) for q in (1, 2, 3)]
    nan = good.copy(order="F")
    nan[3, 3, 3] = np.nan
    return [to_dev(a) for a in (bad[0], good, bad[1], nan, bad[2])]


def hand_over_case(n, maxcy):
    """A context, the members, their solutions and reports alone."""
    g = G.shear_layer_grid(*n, stretched=True)
    p = zline(g, 1e-11)
    p.maxcy = maxcy
    s, rhs = MGSolver(g, p), members(g)
    phi, reps = [torch.zeros_like(f) for f in rhs], []
    for q, f in zip(phi, rhs):
        s.solve(q, f)
        reps.append(s.last_report)
    assert [r.reserved for r in reps] == [0, 1, 0, 1, 0]
    return s, rhs, phi, reps


def assert_batch_equals(s, rhs, phi, reps):
    got = [torch.zeros_like(f) for f in rhs]
    for r, w in zip(s.solve_batch(got, rhs), reps):
        assert (r.status, r.iter, r.reserved) == (w.status, w.iter, w.reserved)
        np.testing.assert_array_equal([r.resid, r.relmax], [w.resid, w.relmax])
    for q, w in zip(got, phi):
        assert torch.equal(q.nan_to_num(), w.nan_to_num())


def test_batch_hands_over_together():
    """Members that need V-cycles get them in one batched loop, with the
    results of their solves alone, beside members that need none; then in
    batches of one and two such members."""
    s, rhs, phi, reps = hand_over_case((16, 8, 64), 12)
    assert_batch_equals(s, rhs, phi, reps)
    n0 = lib().anel_kernel_launch_count()
    assert_batch_equals(s, rhs, phi, reps)
    assert lib().anel_kernel_launch_count() - n0 < 0.5 * sum(r.launches for r in reps)
    for pick in (slice(1, 3), slice(1, 5)):
        assert_batch_equals(s, rhs[pick], phi[pick], reps[pick])
    s.close()


def test_batch_hands_over_without_further_memory():
    """What the V-cycles need has been there since the batch was reserved:
    256x128x128, with less than a member's levels left free."""
    s, rhs, phi, reps = hand_over_case((256, 128, 128), 4)
    assert_batch_equals(s, [rhs[1]] * 5, [phi[1]] * 5, [reps[1]] * 5)
    got = [torch.zeros_like(f) for f in rhs]
    with memory_left(24 << 20):
        out = s.solve_batch(got, rhs)
    assert [(r.status, r.iter) for r in out] == [(r.status, r.iter) for r in reps]
    for q, w in zip(got, phi):
        assert torch.equal(q.nan_to_num(), w.nan_to_num())
    s.close()


def test_batch_within_what_a_serving_bucket_is_charged():
    """Device memory of a context and a batch of eight that hands over,
    against the serving engine's estimate for a bucket's batch solver: 24
    bytes a cell, 16 for each member's and its own FP32 levels, and 64 MB."""
    g = G.shear_layer_grid(256, 256, 256, stretched=True)
    p = zline(g, 1e-30)
    p.maxcy = 4
    rhs = torch.randn(g.ghosted[::-1], dtype=torch.float64, device="cuda")
    phi = [torch.zeros_like(rhs) for _ in range(8)]
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    s = MGSolver(g, p)
    for r in s.solve_batch(phi, [rhs] * 8):
        assert r.status == abi.ERR_NOCONV and r.reserved == 0
    used = before - torch.cuda.mem_get_info()[0]
    s.close()
    assert used <= np.prod(g.ghosted) * (24 + 16 * 9) + (64 << 20)
