"""The forward projector over groups of two to five slices per CTA (xct_plan_set_multislice on)
against the per-slice form (off) and the oracle.  Every slice's samples, weights and per-tile float
sums are the per-slice kernel's up to the order of additions and the tile's side, so both meet the
tiled kernel's bar against the oracle, 5e-6 rel-L2, and each other within twice that."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CASES = [  # nx, ny, px, pa, span, centre offset, slices, angles per CTA
    (82, 165, 90, 24, 180.0, 0.0, 2, 128),     # whole tiles of 83 texels: one and two per side
    (66, 67, 131, 17, 360.0, 2.75, 3, 5),      # a tile of 67 and one texel of the next
    (57, 58, 64, 36, 180.0, 0.0, 4, 128),      # 0 and 90 degrees exactly, off-by-one around 58
    (50, 101, 49, 30, 180.0, -7.5, 5, 7),      # tiles of 51, rays cut by the detector's ends
    (33, 20, 40, 9, 200.0, 0.0, 6, 3),         # 4 + 2, images smaller than a tile
    (120, 75, 100, 21, 180.0, 3.25, 7, 21),    # 4 + 3
    (3, 200, 7, 12, 180.0, 0.0, 9, 128),       # 4 + 5, a strip of three columns
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_grouped_forward_matches_per_slice_and_oracle(gpu_ctx, oracle_lib, case):
    import xct
    O = oracle_lib
    nx, ny, px, pa, span, off, dN, chunk = CASES[case]
    rng = np.random.default_rng(120 + case)
    ang = (np.arange(pa) * (span / pa)).astype(np.float32)
    imgs = rng.uniform(0.0, 1.0, (dN, ny, nx)).astype(np.float32)
    cx = px * 0.5 + off
    plan = xct.OSEMPlan(gpu_ctx, nx, ny, px, ang, 1, 1, center_bin=cx, max_batch=dN)
    d = torch.from_numpy(imgs).cuda()
    out = []
    for ms in (0, chunk):
        plan.set_multislice(ms)
        o = torch.empty((dN, pa, px), device="cuda")
        plan.fwd(d, o)
        out.append(o.cpu().numpy().astype(np.float64))
    for z in range(dN):
        want = O.projection(imgs[z], ang, px, cx=cx)
        norm = np.linalg.norm(want)
        for o in out:
            assert np.linalg.norm(o[z] - want) <= 5e-6 * norm, z
        assert np.linalg.norm(out[0][z] - out[1][z]) <= 1e-5 * norm, z
    plan.close()
