"""The small-problem kernels at the edges of their ranges: just inside and just outside 1.6 million samples a
launch (forward, seen in the launches of OSEM1: one, or a tiled one and its finalize) and 600000 pixels
(backprojection), one slice and ten, against the oracle.  Bars of the small-problem tests: ray sums and ratios
5e-6 rel-L2, the backprojection bit-identical."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CASES = [  # nx, ny, px, pa, ss, centre offset, slices, launches of OSEM1
    (420, 423, 430, 18, 2, 0.0, 1, 1),      # 1598940 samples
    (421, 423, 430, 18, 2, -2.5, 1, 2),     # 1602747
    (200, 100, 210, 16, 2, 1.25, 10, 1),    # 1600000
    (200, 101, 210, 16, 2, 0.0, 10, 2),
    (775, 774, 780, 6, 3, 0.0, 1, 1),       # 599850 pixels
    (776, 774, 780, 6, 3, 0.5, 1, 1),       # 600624
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_small_problem_limits(gpu_ctx, oracle_lib, case):
    import xct
    O = oracle_lib
    nx, ny, px, pa, ss, off, dN, launches = CASES[case]
    rng = np.random.default_rng(170 + case)
    ang = (np.arange(pa) * (180.0 / pa)).astype(np.float32)
    cx = px * 0.5 + off
    imgs = rng.uniform(0.1, 1.0, (dN, ny, nx)).astype(np.float32)
    meas = rng.uniform(0.5, 2.0, (dN, pa, px)).astype(np.float32)
    plan = xct.OSEMPlan(gpu_ctx, nx, ny, px, ang, ss, 1, center_bin=cx, max_batch=dN)
    d_i, d_m = torch.from_numpy(imgs).cuda(), torch.from_numpy(meas).cuda()
    for sub in (0, ss - 1):
        r = torch.zeros((dN, pa, px), device="cuda")
        n0 = xct.launch_count()
        plan.osem1(sub, d_i, d_m, r)
        assert xct.launch_count() - n0 == launches
        x = d_i.clone()
        plan.osem2(sub, x, d_m)
        for z in {0, dN - 1}:
            # a corner ray may sum to just about the ratio's threshold 1e-4: either branch
            p = O.projection(imgs[z], ang, px, cx=cx)
            want = O.osem1(imgs[z], meas[z], ang, ss, sub, cx=cx, order=O.ORDER_GPU)
            got = r[z].cpu().numpy()
            rows = np.arange(sub, sub + pa // ss * ss, ss)
            d = np.where(np.abs(p[rows] - 1.0e-4) < 1.0e-8, 0.0, got[rows].astype(np.float64) - want[rows])
            assert np.linalg.norm(d) <= 5e-6 * np.linalg.norm(want[rows]), (sub, z)
            assert not got[np.setdiff1d(np.arange(pa), rows)].any()
            ref = O.osem2(imgs[z], meas[z], ang, ss, sub, cx=cx, order=O.ORDER_GPU)
            assert np.array_equal(x[z].cpu().numpy(), ref), (sub, z)
    plan.close()
