"""xct_osem_profile (and the XCT_TRACE line, which is made the same way) times the kernels that the call
runs.  A small problem's forward kernel forms the ratio itself: the profiled run launches as many kernels as
the plain call, reports no finalize launch, and -- the small-problem kernels add in a fixed order -- gives
the same bits.  One step larger, the tiled forward kernel and its finalize are reported."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CASES = [(64, 64, 72, 45, 5, 2, True), (33, 61, 50, 20, 3, 1, True), (400, 390, 400, 40, 4, 2, False)]  # ..., ss, slices


@pytest.mark.parametrize("case", range(len(CASES)))
def test_profile_runs_the_calls_kernels(gpu_ctx, case):
    import xct
    nx, ny, px, pa, ss, dN, small = CASES[case]
    it = 2
    ang = (np.arange(pa) * (180.0 / pa)).astype(np.float32)
    plan = xct.OSEMPlan(gpu_ctx, nx, ny, px, ang, ss, it, max_batch=dN)
    sino = (torch.rand((dN, pa, px), generator=torch.Generator().manual_seed(case)) + 0.5).cuda()
    x, y = torch.ones((dN, ny, nx), device="cuda"), torch.ones((dN, ny, nx), device="cuda")
    n0 = xct.launch_count()
    plan.run_device(sino, x)
    torch.cuda.synchronize()
    n1 = xct.launch_count()
    prof = plan.profile(sino, y)
    n2 = xct.launch_count()
    steps = ss * it
    assert n1 - n0 == n2 - n1 == steps * (2 if small else 3)
    assert prof["fwd"]["launches"] == prof["bp"]["launches"] == steps
    assert prof["finalize"]["launches"] == (0 if small else steps)
    assert prof["total"]["launches"] == steps * (2 if small else 3)
    assert prof["fwd"]["ms"] > 0 and prof["bp"]["ms"] > 0 and (prof["finalize"]["ms"] > 0) == (not small)
    if small:
        assert torch.equal(x, y)
    else:
        assert float((x - y).norm() / x.norm()) <= 1e-6
    plan.close()
