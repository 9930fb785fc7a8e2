"""Calls with more slices than a grid's third extent holds (65535): 70000 slices of 4 x 5 pixels, OS-EM and
compressed-sensing OS-EM.  Slices on both sides of the launches' boundary and at the ends get the image
they get in a small call: OS-EM slices are independent; a compressed-sensing slice depends on the stack's first
slice and, over ss * it steps, on as many slices after it (so does the first slice), so a short stack of the
same first eight slices and the same run of slices gives the same images away from its end.  The bar is the forms' against each other over
the steps, 1e-5 of the largest pixel."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

NX, NY, PX, PA, SS, IT, DN = 4, 5, 7, 6, 2, 2, 70000


@pytest.mark.parametrize("cs", [False, True])
def test_more_slices_than_a_grid_extent(gpu_ctx, cs):
    import xct
    ang = (np.arange(PA) * (180.0 / PA)).astype(np.float32)
    sino = (torch.rand((DN, PA, PX), generator=torch.Generator().manual_seed(9)) + 0.5).cuda()

    def run(s):
        plan = xct.OSEMPlan(gpu_ctx, NX, NY, PX, ang, SS, IT, max_batch=len(s))
        x = torch.ones((len(s), NY, NX), device="cuda")
        if cs:
            plan.cs_run_device(s, x, cs_lambda=1.0e-3)
        else:
            plan.run_device(s, x)
        torch.cuda.synchronize()
        plan.close()
        return x.cpu().numpy()

    whole = run(sino)
    assert np.isfinite(whole).all()
    steps, head = SS * IT, 8
    for first in (1, 65500, DN - 60):
        last = min(first + 60, DN)
        part = run(torch.cat([sino[:head], sino[first:last]]).contiguous())
        keep = last - first - (steps if cs and last < DN else 0)
        a, b = whole[first:first + keep], part[head:head + keep]
        assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max(), first
