"""The exact adjoint's forms -- scatter with one or two slices per CTA on tiles of 16, 32, 44 and 64
texels, gather over four, eight and ten slices -- on rays of both signs whose magnitudes span the
fixed-point levels (down to 2^-17 of the largest), with zero rays, an odd size and an off-centre axis.
Each contribution rounds by at most 2^-16 of its ray's value in the scatter form and as a float in the
gather form, so the result stays within 1e-5 rel-L2 of the oracle's sum with the same float32 coordinates;
the forms of one input agree within twice that."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CASES = [  # nx, ny, px, pa, span, centre offset, slices
    (1, 1, 3, 5, 180.0, 0.0, 1),
    (15, 33, 20, 40, 180.0, 0.0, 1),       # tiles of 16, two windows of angles
    (130, 97, 170, 33, 360.0, 2.25, 2),    # rays longer than the image, a window of one angle
    (300, 310, 280, 12, 180.0, -4.5, 3),   # rays off the detector
    (700, 650, 720, 6, 180.0, 0.0, 2),
    (1000, 900, 1010, 4, 180.0, 0.0, 1),   # 0 and 90 degrees exactly, the largest tiles
    (64, 50, 70, 50, 200.0, 1.5, 4),
    (93, 61, 100, 47, 180.0, -3.75, 10),
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_adjoint_forms_match_oracle(gpu_ctx, oracle_lib, case):
    import xct
    O = oracle_lib
    nx, ny, px, pa, span, off, dN = CASES[case]
    rng = np.random.default_rng(140 + case)
    ang = (np.arange(pa) * (span / pa)).astype(np.float32)
    y = (2.0 ** rng.uniform(-17, 0, (dN, pa, px)) * rng.choice([-1.0, 0.0, 1.0], (dN, pa, px), p=[0.45, 0.1, 0.45])).astype(np.float32)
    cx = px * 0.5 + off
    plan = xct.OSEMPlan(gpu_ctx, nx, ny, px, ang, 1, 1, center_bin=cx, max_batch=dN)
    d = torch.from_numpy(y).cuda()
    got = []
    for off_by_hand in (False, True):
        if off_by_hand:
            plan.set_multislice(0)
        a = torch.full((dN, ny, nx), float("nan"), device="cuda")
        plan.adj(d, a)
        got.append(a.cpu().numpy().astype(np.float64))
    for z in range(dN):
        want = O.adjoint(y[z], ang, nx, ny, cx=cx).astype(np.float64)
        norm = max(np.linalg.norm(want), 1e-30)
        for g in got:
            assert np.linalg.norm(g[z] - want) <= 1e-5 * norm, z
        assert np.linalg.norm(got[0][z] - got[1][z]) <= 2e-5 * norm, z
    plan.close()
