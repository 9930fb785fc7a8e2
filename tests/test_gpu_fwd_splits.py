"""The divisions of the forward launches that a plan keeps.  A call's division depends on its slices, its
angles and the plan's cap on angles a pass; a plan that has served many such calls, more than it keeps, gives
each the ray sums of a plan that serves nothing else (the same samples and partial sums, whose double sums
meet in any order: 1e-6 rel-L2).  And finding the division is no part of a repeated call: a default plan's
forward call costs the host at most 1.3 times one with its tile set by hand, which has nothing to find (both
are two launches; measured 1.0, and 1.7 when every call divided anew)."""
import time

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def test_kept_divisions_serve_their_calls_only(gpu_ctx):
    import xct
    nx, ny, px, pa, ss, most = 300, 270, 310, 101, 4, 9
    ang = (np.arange(pa) * (180.0 / pa)).astype(np.float32)
    kw = dict(center_bin=151.5, subset_mode=xct.SUBSETS_COVER, max_batch=most)
    gen = torch.Generator().manual_seed(5)
    img = (torch.rand((most, ny, nx), generator=gen) + 0.1).cuda()
    meas = (torch.rand((most, pa, px), generator=gen) + 0.5).cuda()
    plan = xct.OSEMPlan(gpu_ctx, nx, ny, px, ang, ss, 1, **kw)

    def calls(p, dN):
        out = []
        f = torch.empty((dN, pa, px), device="cuda")
        p.fwd(img[:dN].contiguous(), f)
        out.append(f)
        for sub in (0, ss - 1):  # 26 and 25 rows
            r = torch.zeros((dN, pa, px), device="cuda")
            p.osem1(sub, img[:dN].contiguous(), meas[:dN].contiguous(), r)
            out.append(r)
        return [o.cpu().numpy().astype(np.float64) for o in out]

    for cap in (128, 6):
        plan.set_multislice(cap)
        for dN in (9, 4, 1, 8, 5, 2, 3, 9, 1):
            fresh = xct.OSEMPlan(gpu_ctx, nx, ny, px, ang, ss, 1, **kw)
            fresh.set_multislice(cap)
            for a, b in zip(calls(plan, dN), calls(fresh, dN)):
                assert np.linalg.norm(a - b) <= 1e-6 * np.linalg.norm(b), (cap, dN)
            fresh.close()
    plan.close()


def test_division_is_found_once(gpu_ctx):
    import xct
    n, pa = 192, 67
    ang = (np.arange(pa) * (180.0 / pa)).astype(np.float32)
    img, out = torch.rand((2, n, n), device="cuda"), torch.empty((2, pa, n), device="cuda")
    us = []
    for by_hand in (False, True):
        plan = xct.OSEMPlan(gpu_ctx, n, n, n, ang, 1, 1, max_batch=2)
        if by_hand:
            plan.set_tuning(44, 16)
        plan.fwd(img, out)
        n0 = xct.launch_count()
        plan.fwd(img, out)
        assert xct.launch_count() - n0 == 2
        best = []
        for _ in range(80):  # short bursts: the queue never fills
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            for _ in range(10):
                plan.fwd(img, out)
            best.append(time.perf_counter() - t0)
        us.append(min(best) * 1e5)
        torch.cuda.synchronize()
        plan.close()
    assert us[0] <= 1.3 * us[1], us
