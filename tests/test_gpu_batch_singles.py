"""Single slices of a batch plan on the large forward tiles (163 texels, one CTA per SM) against each slice
alone in its own plan with its tile set by hand.  The samples are the same and only the partial sums that
meet in double differ, as in the batch plan's other forms: their bar, 1e-6 rel-L2.  Sizes at the tile's edge
(n + 1 = 7 * 163 and one more), non-square, an off-centre axis, subsets that do not divide the angles,
more angles per subset than one chunk (128); and the same after the autotuner chose."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

SHAPES = [  # nx, ny, px, angles, subsets' cover mode, centre offset
    (1140, 1141, 1140, 270, False, 0.0),
    (977, 650, 990, 271, True, 2.25),
    (163, 900, 301, 262, False, -3.5),
]


@pytest.mark.parametrize("tune", [False, True])
def test_large_single_slices(gpu_ctx, tune):
    import xct
    geoms, sinos, want = [], [], []
    for j, (nx, ny, px, pa, cover, off) in enumerate(SHAPES):
        ang = (np.arange(pa) * (180.0 / pa)).astype(np.float32)
        mode = xct.SUBSETS_COVER if cover else xct.SUBSETS_REF
        geoms.append(xct.make_geom(nx, ny, px, ang, 2, 1, center_bin=px * 0.5 + off, subset_mode=mode))
        sino = torch.rand((pa, px), generator=torch.Generator().manual_seed(j)).cuda() + 0.5
        sinos.append(sino)
        plan = xct.OSEMPlan(gpu_ctx, nx, ny, px, ang, 2, 1, center_bin=px * 0.5 + off, subset_mode=mode, max_batch=1)
        plan.set_tuning(76, 64)
        img = torch.ones((1, ny, nx), device="cuda")
        plan.run_device(sino[None].contiguous(), img)
        want.append(img[0].cpu().numpy().astype(np.float64))
        plan.close()
    bp = xct.BatchPlan(gpu_ctx, geoms, 1)
    if tune:
        bp.autotune(force=True)
    for replay in range(2):
        imgs = [torch.ones((s[1], s[0]), device="cuda") for s in SHAPES]
        bp.run(sinos, imgs)
        for k, x in enumerate(imgs):
            got = x.cpu().numpy().astype(np.float64)
            assert np.linalg.norm(got - want[k]) <= 1e-6 * np.linalg.norm(want[k]), (replay, k)
    bp.close()
