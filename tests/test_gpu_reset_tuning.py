"""Choices made by hand can be taken back.  After set_tuning and set_multislice, on or off, reset_tuning leaves the
plan as it was created: the same reported values, the same launches per call, and for a small problem, whose
kernels add in a fixed order, the same bits."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [(64, 30, 5, 3), (300, 60, 4, 10), (740, 14, 2, 10)])  # n, angles, subsets, slices
def test_reset_restores_the_plans_own_choices(gpu_ctx, case):
    import xct
    n, pa, ss, dN = case
    ang = (np.arange(pa) * (180.0 / pa)).astype(np.float32)
    plan = xct.OSEMPlan(gpu_ctx, n, n, n, ang, ss, 1, max_batch=dN)
    sino = (torch.rand((dN, pa, n), generator=torch.Generator().manual_seed(n)) + 0.5).cuda()

    def state():
        x, a = torch.ones((dN, n, n), device="cuda"), torch.empty((dN, n, n), device="cuda")
        n0 = xct.launch_count()
        plan.run_device(sino, x)
        n1 = xct.launch_count()
        plan.adj(sino, a)
        torch.cuda.synchronize()
        return (plan.tuning(), plan.multislice(), n1 - n0, xct.launch_count() - n1), x

    own, want = state()
    for change in (lambda: plan.set_tuning(44, 5), lambda: plan.set_multislice(0), lambda: plan.set_multislice(9),
                   lambda: (plan.set_multislice(0), plan.set_tuning(92, 16))):
        change()
        assert state()[0] != own
        plan.reset_tuning()
        got, x = state()
        assert got == own
        if n == 64:
            assert torch.equal(x, want)
        else:
            assert float((x - want).norm() / want.norm()) <= 1e-6
    plan.close()
