"""What a context does after a call that failed: an allocation that the
device cannot meet is an error of that call alone, and leaves no state that
later calls would take for that of a call that succeeded."""
import contextlib

import numpy as np
import pytest

from anelastic_solve_b200 import abi, shear
from anelastic_solve_b200 import grid as G
from anelastic_solve_b200._lib import AnelError
from anelastic_solve_b200.mg import MGSolver
from anelastic_solve_b200.ns import NSSolver

from .helpers import compatible, field, levels_for, mg_params
from .test_mg_batch import to_dev, to_host

pytestmark = pytest.mark.gpu


def zline(g, tol):
    return mg_params(g, levels=levels_for(g)[:2] + (1,), mode=abi.MODE_METRIC, smoother=abi.SMOOTHER_ZLINE,
                     maxcy=60, tolmax=tol, stop=abi.STOP_RESID, precision=abi.PREC_MIXED)


def refused_batch(s, phi, rhs, members):
    """A batch of more members than the device has memory for (every member
    the same two arrays: the call fails before its first launch)."""
    with pytest.raises(AnelError) as e:
        s.solve_batch([phi] * members, [rhs] * members)
    assert e.value.code == abi.ERR_CUDA


def test_solve_after_a_batch_without_memory():
    """64^3 by V-cycles: 2 MB of FP32 levels a member."""
    g = G.shear_layer_grid(64, 64, 64, stretched=True)
    rhs = to_dev(compatible(field(g, np.random.default_rng(1)), g, abi.MODE_METRIC))
    s = MGSolver(g, zline(g, 1e-10))
    want, got = rhs * 0.0, rhs * 0.0
    s.solve(want, rhs)
    refused_batch(s, got, rhs, 200_000)
    s.solve(got, rhs)
    assert s.last_report.status == abi.OK
    np.testing.assert_array_equal(to_host(got), to_host(want))
    (rep,) = s.solve_batch([got], [rhs])
    assert rep.status == abi.OK and rep.iter == 0
    s.close()


def test_direct_solve_after_a_batch_without_memory():
    """512x256x512: 0.26 MB of partial sums a member, so a batch of 800 000
    fails at the direct solve's first buffer; the buffers that it had before,
    for one member and for two, go on."""
    import torch

    g = G.shear_layer_grid(512, 256, 512, stretched=True)
    gen = torch.Generator("cuda").manual_seed(1)
    rhs = torch.zeros(g.ghosted[::-1], dtype=torch.float64, device="cuda")
    f = torch.randn(g.shape[::-1], generator=gen, dtype=torch.float64, device="cuda")
    dz = torch.from_numpy(g.z.dxc[1:-1].copy()).cuda()
    rhs[1:-1, 1:-1, 1:-1] = f - (f.mean(dim=(1, 2)) * dz).sum() / dz.sum()
    s = MGSolver(g, zline(g, 1e-11))
    want = torch.zeros_like(rhs)
    s.solve(want, rhs)
    assert s.last_report.reserved == 1
    for reserved in (1, 2):
        if reserved == 2:
            two = [torch.zeros_like(rhs) for _ in range(2)]
            s.solve_batch(two, [rhs, rhs])
        got = torch.zeros_like(rhs)
        refused_batch(s, got, rhs, 800_000)
        s.solve(got, rhs)
        assert s.last_report.status == abi.OK and s.last_report.reserved == 1
        assert torch.equal(got, want)
    got = [torch.zeros_like(rhs) for _ in range(2)]
    for rep in s.solve_batch(got, [rhs, rhs]):
        assert rep.status == abi.OK
    assert torch.equal(got[0], want) and torch.equal(got[1], want)
    s.close()


@contextlib.contextmanager
def memory_left(nbytes):
    """All device memory but nbytes is taken."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - nbytes, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        hog.untyped_storage().resize_(0)
        torch.cuda.empty_cache()


def stepper(g, seed, **phys):
    f = shear.shear_layer_fields(g, amp=1e-2, seed=seed)
    kw = dict(Re=1000.0, Pr=1.0, g=-0.1, cfl=0.5, dtmax=1e9, ew=1, scal1_on=0)
    s = NSSolver(g, zline(g, 1e-11), abi.make_ns_params(**{**kw, **phys}))
    s.set_fields({k: f[k] for k in ("u", "v", "w", "p", "rho", "scal1", "r", "densityBG")})
    s.project()
    return s


FIELDS = ("u", "v", "w", "p", "rho")
# 256x128x128: a field of 36 MB; less than one is left free where a call is
# to fail, and the kernels that it launches have been loaded by then
GRID, LEFT = (256, 128, 128), 24 << 20


def test_a_set_up_that_ran_out_of_memory_is_taken_up_again():
    """The plane statistics' arrays, a small one and then two of the size of
    a field: a call that could not have them all fails, and a step with
    memory back equals that of a context that never lacked any."""
    g = G.shear_layer_grid(*GRID, stretched=True)
    a, b = stepper(g, 1), stepper(g, 1)
    for s in (a, b):
        s.set_diagnostics(True)
    a.step(1)
    with memory_left(LEFT), pytest.raises(AnelError) as e:
        b.compute_diagnostics()
    assert e.value.code == abi.ERR_CUDA
    b.step(1)
    want, got = a.get_fields(FIELDS), b.get_fields(FIELDS)
    for k in FIELDS:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    want, got = a.diagnostics(), b.diagnostics()
    for k, v in want.items():
        np.testing.assert_array_equal(got[k], v, err_msg=k)
    a.close()
    b.close()


def failed_cohort(members):
    with memory_left(LEFT), pytest.raises(AnelError) as e:
        NSSolver.step_cohort(members, 1)
    assert e.value.code == abi.ERR_CUDA


def test_time_step_after_a_cohort_step_that_failed_at_its_end():
    """The second member's statistics find no memory after the fields have
    been advanced and before the cohort's divergence pass: the first member's
    next time step comes from the fields it has now."""
    g = G.shear_layer_grid(*GRID, stretched=True)
    ms = [stepper(g, seed) for seed in (1, 2)]
    ms[0].set_diagnostics(True)
    before = NSSolver.step_cohort(ms, 2)[0]
    ms[1].set_diagnostics(True)
    failed_cohort(ms)
    ref = stepper(g, 1)
    ref.set_fields(ms[0].get_fields(FIELDS + ("scal1",)))
    want = ref.step(1)
    got = ms[0].step(1)
    assert got.nstep == before.nstep + 2 and got.dt == want.dt != before.dt
    for s in (*ms, ref):
        s.close()


def test_column_factors_after_a_cohort_step_that_failed_at_its_start():
    """The second member's dynamic model finds no memory before the members'
    Crank-Nicolson factors are made for their new time steps: the first
    member's next step makes them."""
    g = G.shear_layer_grid(*GRID, stretched=True)
    kw = dict(les=True, Re=5e4, models=(abi.MODEL_DSM,) * 3)
    ref, *ms = (stepper(g, seed, **kw) for seed in (1, 1, 2))
    for s in (ref, ms[0]):
        s.step(1)
    failed_cohort(ms)
    ref.step(1)
    ms[0].step(1)
    want, got = ref.get_fields(FIELDS), ms[0].get_fields(FIELDS)
    for k in FIELDS:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    for s in (*ms, ref):
        s.close()
