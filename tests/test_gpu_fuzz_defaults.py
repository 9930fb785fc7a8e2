"""Seeded random geometries through plans as they are created -- no tile and no switch set by hand, so that
the small-problem kernels, the runs, the groups of two to five slices and the adjoint's forms are what the
sizes make them -- against the oracle: 17..420 pixels a side, 16..460 bins, 5..110 angles over 180, 200 or 360
degrees, sorted or not, 1..9 subsets in either mode, an off-centre axis, 1..13 slices.

Bars, as for the tiled kernels with tiles by hand: ratio rows 5e-6 rel-L2, other rows untouched; OSEM2 of given
ratios and the FBP backprojection bit-identical; the adjoint 1e-5 rel-L2 of the float64 one."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

SLICES = [1, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 13]


@pytest.mark.parametrize("seed", range(len(SLICES)))
def test_default_plans_on_random_geometries(gpu_ctx, oracle_lib, seed):
    import xct
    O = oracle_lib
    rng = np.random.default_rng(3000 + seed)
    dN = SLICES[seed]
    nx, ny = (int(round(np.exp(rng.uniform(np.log(17), np.log(420))))) for _ in range(2))
    px, pa = int(rng.integers(16, 461)), int(rng.integers(5, 111))
    ss = int(rng.integers(1, min(9, pa) + 1))
    cover = bool(rng.integers(0, 2))
    ang = rng.uniform(0.0, float(rng.choice([180.0, 200.0, 360.0])), pa).astype(np.float32)
    if rng.uniform() < 0.5:
        ang = np.sort(ang)
    cx = px * 0.5 + float(rng.uniform(-8.0, 8.0))
    imgs = rng.uniform(0.05, 1.0, (dN, ny, nx)).astype(np.float32)
    meas = rng.uniform(0.5, 2.0, (dN, pa, px)).astype(np.float32)
    where = "seed %d: nx %d ny %d px %d pa %d ss %d cover %d cx %.3f slices %d" % (seed, nx, ny, px, pa, ss, cover, cx, dN)
    plan = xct.OSEMPlan(gpu_ctx, nx, ny, px, ang, ss, 1, center_bin=cx, max_batch=dN,
                        subset_mode=xct.SUBSETS_COVER if cover else xct.SUBSETS_REF)
    d_i, d_m = torch.from_numpy(imgs).cuda(), torch.from_numpy(meas).cuda()
    look = sorted({0, dN // 2, dN - 1})
    proj = {z: O.projection(imgs[z], ang, px, cx=cx) for z in look}
    fwd = torch.empty((dN, pa, px), device="cuda")
    plan.fwd(d_i, fwd)
    for z in look:
        assert np.linalg.norm(fwd[z].cpu().numpy() - proj[z]) <= 5e-6 * max(np.linalg.norm(proj[z]), 1e-30), where
    for sub in sorted({0, ss - 1}):
        rows = np.arange(sub, pa if cover else sub + pa // ss * ss, ss)
        r = torch.full((dN, pa, px), -7.0, device="cuda")
        plan.osem1(sub, d_i, d_m, r)
        x = d_i.clone()
        plan.osem2(sub, x, d_m)
        for z in look:
            p, m = proj[z][rows].astype(np.float64), meas[z][rows]
            want = np.where(p < 1.0e-4, m, m / np.where(p < 1.0e-4, 1.0, p))
            got = r[z].cpu().numpy()
            d = np.where(np.abs(p - 1.0e-4) < 1.0e-8, 0.0, got[rows] - want)  # either branch of the ratio there
            assert np.linalg.norm(d) <= 5e-6 * np.linalg.norm(want), where
            assert np.all(got[np.setdiff1d(np.arange(pa), rows)] == -7.0), where
            ref = O.osem2(imgs[z], meas[z], ang, ss, sub, cx=cx, order=O.ORDER_GPU)
            assert np.array_equal(x[z].cpu().numpy(), ref), where
    f = torch.empty((dN, ny, nx), device="cuda")
    plan.fbp_backproject(d_m, f)
    a = torch.empty((dN, ny, nx), device="cuda")
    plan.adj(d_m, a)
    for z in look:
        assert np.array_equal(f[z].cpu().numpy(), O.bp_fbp(meas[z], ang, nx, ny, cx=cx)), where
        want = O.adjoint(meas[z], ang, nx, ny, cx=cx, dtype=np.float64)
        assert np.linalg.norm(a[z].cpu().numpy() - want) <= 1e-5 * np.linalg.norm(want), where
    plan.close()
