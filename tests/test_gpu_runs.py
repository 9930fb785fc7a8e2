"""The forward projector's large tiles and its division of (tile, angle) units into runs, one per CTA:
against the chunked per-slice kernel (a plan with its tile set by hand), which samples the same points and
differs only in which partial sums meet in double.  A lane adds at most 163 * sqrt(2) / 4 + 1 samples of a
tile (60 * sqrt(2) / 4 + 1 in the chunked kernel), two roundings each, and one more joins a ray's lanes: 119
and 46 roundings of 2^-24 of sums of positive terms, and one of the result on either side.  The bar is their
sum, 167 * 2^-24 = 1.0e-5 of the ray sum.

Sizes: one tile exactly and one texel more (base texels are -1 .. n-1) for the sides of one to five slices,
fewer units than CTAs, as many tiles as CTAs, more angles than one pass of a CTA (128), tiles whose rays
miss a narrow detector, an off-centre axis, groups of five and four."""
import numpy as np
import pytest
import torch

import xct

pytestmark = pytest.mark.gpu

CASES = [
    # nx, ny, px, pa, ss, slices, center, most angles a pass
    (162, 162, 162, 20, 2, 1, None, 128),
    (163, 230, 170, 21, 2, 1, None, 128),
    (700, 690, 711, 40, 2, 1, 350.0, 128),
    (2000, 1970, 2000, 6, 3, 1, None, 128),
    (114, 115, 120, 30, 1, 2, None, 128),
    (900, 400, 301, 26, 1, 2, 100.5, 128),
    (92, 93, 92, 3, 1, 3, None, 128),
    (640, 640, 640, 140, 1, 3, None, 9),
    (82, 83, 90, 24, 2, 4, None, 128),
    (1030, 1000, 1030, 25, 1, 8, None, 128),
    (74, 75, 80, 10, 1, 5, None, 128),
    (300, 290, 310, 22, 2, 10, 160.0, 128),
    (130, 5, 140, 9, 1, 10, None, 128),
]


@pytest.mark.parametrize("case", CASES)
def test_runs_match_chunks(gpu_ctx, case):
    nx, ny, px, pa, ss, dN, center, cap = case
    ang = (np.arange(pa) * (180.0 / pa)).astype(np.float32)
    plan = xct.OSEMPlan(gpu_ctx, nx, ny, px, ang, ss, 1, center_bin=center, max_batch=dN)
    hand = xct.OSEMPlan(gpu_ctx, nx, ny, px, ang, ss, 1, center_bin=center, max_batch=dN)
    hand.set_tuning(60, 7)
    plan.set_multislice(cap)  # the grouped form whatever the size
    img = torch.rand((dN, ny, nx), generator=torch.Generator().manual_seed(nx + pa)).cuda() + 0.1
    got, want = (torch.empty((dN, pa, px), device="cuda") for _ in range(2))
    plan.fwd(img, got)
    hand.fwd(img, want)
    torch.cuda.synchronize()
    err = ((got - want).abs() / want.abs().clamp(min=1.0e-3)).max().item()
    assert err <= 1.0e-5, "%s: %.3e" % (case, err)
    plan.fwd(img, want)  # the accumulator is left cleared
    err = ((got - want).abs() / want.abs().clamp(min=1.0e-3)).max().item()
    assert err <= 1.0e-5, "%s again: %.3e" % (case, err)
    plan.close()
    hand.close()
