"""Images with more than 4096 forward tiles a slice, where a launch takes a CTA per tile and chunk of angles
instead of runs, on the large tiles: one slice and four, against the plan with its tile set by hand (the
same samples; partial sums of longer rays meet in double: the runs' bar, 1.0e-5 of the ray sum)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CASES = [  # nx, ny, bins, slices: tiles of 163 and of 83 texels
    (16384, 6700, 700, 1),   # 101 x 42
    (16383, 1750, 640, 4),   # 198 x 22
]


@pytest.mark.parametrize("case", CASES)
def test_more_tiles_than_runs_can_weigh(gpu_ctx, case):
    import xct
    nx, ny, px, dN = case
    ang = np.asarray([0.0, 37.5, 90.0, 140.25], np.float32)
    gen = torch.Generator(device="cuda").manual_seed(ny)
    img = torch.rand((dN, ny, nx), device="cuda", generator=gen) + 0.1
    out = []
    for by_hand in (False, True):
        plan = xct.OSEMPlan(gpu_ctx, nx, ny, px, ang, 1, 1, max_batch=dN)
        if by_hand:
            plan.set_tuning(92, 3)
        o = torch.empty((dN, len(ang), px), device="cuda")
        plan.fwd(img, o)
        torch.cuda.synchronize()
        out.append(o)
        plan.close()
    assert float(out[1].min()) > 0.0
    err = float(((out[0] - out[1]).abs() / out[1]).max())
    assert err <= 1.0e-5, err
