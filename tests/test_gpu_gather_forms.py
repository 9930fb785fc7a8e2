"""The gather adjoint over four, eight and ten slices, and beside leftover slices, at sizes that the choice of
forms sends to it: against the oracle on rays of both signs spanning 2^-17 of the largest, at odd sizes and
off-centre axes, with rays off the detector; and its epilogue (a gradient step, base + scale * A^T y).

That the gather ran is asserted by what only it does: a texel's sum depends on the rays that meet the
texel and on no other, so making one ray 2^20 times larger leaves every texel away from that ray the same
bits.  The scatter's fixed-point scale follows the largest ray of a tile's window, so its bits change there.

Bars: float sums with the oracle's float32 coordinates, 1e-5 rel-L2, and the gradient step against the
per-slice form 1e-6, as in the other adjoint tests."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CASES = [  # nx, ny, px, angles, span, centre offset, slices, slices that the gather takes
    (301, 277, 310, 21, 180.0, 0.0, 4, 4),
    (200, 200, 150, 33, 360.0, -3.25, 4, 4),
    (330, 301, 400, 17, 200.0, 5.5, 8, 8),
    (401, 390, 401, 16, 180.0, 0.0, 10, 10),
    (311, 305, 320, 18, 180.0, 2.75, 9, 8),
    (310, 290, 300, 9, 180.0, 0.0, 12, 12),
]


def _plan(xct, ctx, case):
    nx, ny, px, pa, span, off, dN, _ = case
    ang = (np.arange(pa) * (span / pa)).astype(np.float32)
    return ang, px * 0.5 + off, xct.OSEMPlan(ctx, nx, ny, px, ang, 1, 1, center_bin=px * 0.5 + off, max_batch=dN)


@pytest.mark.parametrize("case", range(len(CASES)))
def test_gather_matches_oracle(gpu_ctx, oracle_lib, case):
    import xct
    nx, ny, px, pa, span, off, dN, most = CASES[case]
    ang, cx, plan = _plan(xct, gpu_ctx, CASES[case])
    rng = np.random.default_rng(160 + case)
    y = (2.0 ** rng.uniform(-17, 0, (dN, pa, px)) * rng.choice([-1.0, 0.0, 1.0], (dN, pa, px), p=[0.45, 0.1, 0.45])).astype(np.float32)

    def adj(v):
        a = torch.full((dN, ny, nx), float("nan"), device="cuda")
        plan.adj(torch.from_numpy(v).cuda(), a)
        return a.cpu().numpy()

    got = adj(y)
    for z in range(dN):
        want = oracle_lib.adjoint(y[z], ang, nx, ny, cx=cx).astype(np.float64)
        assert np.linalg.norm(got[z] - want) <= 1e-5 * np.linalg.norm(want), z
    th, X = pa // 3, int(cx) + 7  # the ray made large, and the texels it does not meet
    phi = float(ang[th]) * np.pi / 180.0
    u = (np.arange(nx)[None, :] - nx * 0.5) * np.cos(phi) - (np.arange(ny)[:, None] - ny * 0.5) * np.sin(phi) + cx
    away = np.abs(u - X) > 4.0
    large = y.copy()
    large[:, th, X] = 2.0 ** 20
    for by_hand in (False, True):
        if by_hand:
            plan.set_multislice(0)  # every slice scattered alone
        a, b = adj(y), adj(large)
        same = [np.array_equal(a[z][away], b[z][away]) for z in range(dN)]
        assert same == [not by_hand and z < most for z in range(dN)], (by_hand, same)
    plan.close()


@pytest.mark.parametrize("case", [0, 2, 3])
def test_gather_gradient_step(gpu_ctx, case):
    import xct
    from xct import phantom as P
    nx, ny, px, pa, span, off, dN, _ = CASES[case]
    ang, cx = (np.arange(24) * (180.0 / 24)).astype(np.float32), px * 0.5 + off
    plan = xct.OSEMPlan(gpu_ctx, nx, ny, px, ang, 4, 2, center_bin=cx, max_batch=dN)
    m = max(nx, ny)
    imgs = np.stack([P.rasterize_ellipses(P.ellipse_params(m, 5, z, axes=(3, m / 4)), m, m)[:ny, :nx] for z in range(dN)])
    plan.set_lipschitz(plan.power_iteration(trials=5, work_group=64))
    meas = torch.empty((dN, 24, px), device="cuda")
    plan.fwd(torch.from_numpy(np.ascontiguousarray(imgs, np.float32)).cuda(), meas)
    out = []
    for by_hand in (False, True):
        if by_hand:
            plan.set_multislice(0)
        x = torch.zeros((dN, ny, nx), device="cuda")
        plan.fista_run_device(meas, x, flags=xct.FISTA_ADJOINT | xct.FISTA_UPDATE_X)
        out.append(x.cpu().numpy().astype(np.float64))
    assert np.isfinite(out[0]).all() and np.abs(out[0]).max() > 0
    assert np.linalg.norm(out[0] - out[1]) <= 1e-6 * np.linalg.norm(out[1])
    plan.close()
