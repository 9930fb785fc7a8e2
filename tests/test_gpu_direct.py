"""The small-problem OS-EM kernels (complete ray sums per launch, one pixel per thread) against
the oracle and against the tiled kernels, which a plan with tiles chosen by hand keeps at every
size.  A ray sum adds the same float samples in another order (float within a lane, then
double), so the bar is the tiled kernel's own against the oracle, 5e-6 rel-L2; OSEM2 adds its bins
in angle order and is bit-identical."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CASES = [  # nx, ny, px, pa, ss, centre offset, slices, fetch mode, cover
    (1, 1, 1, 4, 2, 0.0, 1, 0, 0),           # one texel
    (5, 3, 9, 7, 3, 0.25, 2, 0, 1),          # fewer samples than lanes, a partial ray group
    (33, 31, 40, 19, 4, -1.5, 3, 1, 0),      # odd sizes, an odd slice left over, averaged fetch
    (64, 64, 64, 36, 4, 0.0, 1, 0, 0),       # 0 and 90 degrees exactly
    (130, 70, 97, 30, 4, 3.375, 5, 0, 1),    # rays longer than the image is high
    (700, 650, 720, 18, 2, 0.0, 1, 0, 0),    # the largest size of the forward kernel's range
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_direct_steps_match_oracle_and_tiles(gpu_ctx, oracle_lib, case):
    import xct
    O = oracle_lib
    nx, ny, px, pa, ss, off, dN, fetch, cover = CASES[case]
    rng = np.random.default_rng(90 + case)
    ang = (np.arange(pa) * (180.0 / pa)).astype(np.float32)
    imgs = rng.uniform(0.0, 1.0, (dN, ny, nx)).astype(np.float32)
    meas = rng.uniform(-0.1, 2.0, (dN, pa, px)).astype(np.float32)
    cx = px * 0.5 + off
    plan = xct.OSEMPlan(gpu_ctx, nx, ny, px, ang, ss, 1, center_bin=cx, fetch_mode=fetch, max_batch=dN,
                        subset_mode=xct.SUBSETS_COVER if cover else xct.SUBSETS_REF)
    tiled = xct.OSEMPlan(gpu_ctx, nx, ny, px, ang, ss, 1, center_bin=cx, fetch_mode=fetch, max_batch=dN,
                         subset_mode=xct.SUBSETS_COVER if cover else xct.SUBSETS_REF)
    tiled.set_tuning(44, 16)
    d_i, d_m = torch.from_numpy(imgs).cuda(), torch.from_numpy(meas).cuda()
    raw = [torch.empty((dN, pa, px), device="cuda") for _ in range(2)]
    plan.fwd(d_i, raw[0])
    tiled.fwd(d_i, raw[1])
    for z in range(dN):
        want = O.projection(imgs[z], ang, px, cx=cx)
        for r in raw:
            assert np.linalg.norm(r[z].cpu().numpy() - want) <= 5e-6 * max(np.linalg.norm(want), 1e-30), z
    for sub in (0, ss - 1):
        r = torch.zeros((dN, pa, px), device="cuda")
        t = torch.zeros((dN, pa, px), device="cuda")
        plan.osem1(sub, d_i, d_m, r)
        tiled.osem1(sub, d_i, d_m, t)
        r, t = r.cpu().numpy().astype(np.float64), t.cpu().numpy().astype(np.float64)
        rows = (pa - sub + ss - 1) // ss if cover else pa // ss
        other = np.ones(pa, bool)
        other[sub:sub + rows * ss:ss] = False
        assert not r[:, other].any()
        # ray sums within rounding of the threshold 1e-4 may choose either branch of the ratio
        near = np.abs(raw[1].cpu().numpy() - 1.0e-4) < 1e-9
        d = np.where(near, 0.0, r - t)
        assert np.linalg.norm(d) <= 5e-6 * np.linalg.norm(t)
        d_r = torch.from_numpy(rng.uniform(0.5, 1.5, (dN, pa, px)).astype(np.float32)).cuda()
        x, y = d_i.clone(), d_i.clone()
        plan.osem2(sub, x, d_r)
        tiled.osem2(sub, y, d_r)
        assert torch.equal(x, y)
        for z in (0, dN - 1):
            want = O.osem2(imgs[z], d_r[z].cpu().numpy(), ang, ss, sub, cx=cx, order=O.ORDER_GPU)
            assert np.array_equal(x[z].cpu().numpy(), want), (sub, z)
    plan.close()
    tiled.close()
