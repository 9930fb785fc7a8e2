"""The FBP backprojection's slice groups on images that do not fill the GPU.  Three slices of 400^2 (169 tiles for 152
SMs) may not take longer than four: a pair and a single slice one after the other are two launches of about
a CTA's own time each (1.22 of four slices' time), three singles in one launch are not (0.95).  Eight slices
of 768^2 (576 tiles, 456 places for eight-slice CTAs) may not take more than 1.83 of four: the rows of tiles go from
the middle outwards, so that the CTAs of the second round are those with the least to do (1.75; 1.90 from the top
down).  The images are the same bits however the slices are grouped."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,few,many,limit", [(400, 4, 3, 1.05), (768, 4, 8, 1.83)])
def test_more_slices_no_relative_loss(gpu_ctx, n, few, many, limit):
    import xct
    pa = n // 2
    ang = (np.arange(pa) * (180.0 / pa)).astype(np.float32)
    most = max(few, many)
    y = torch.rand((most, pa, n), generator=torch.Generator().manual_seed(n)).cuda()
    ms, imgs = {}, {}
    for k in (few, many, 1):
        plan = xct.OSEMPlan(gpu_ctx, n, n, n, ang, 6, 1, max_batch=k)
        img = torch.empty((k, n, n), device="cuda")
        d = y[:k].contiguous()
        best = []
        for _ in range(12):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            e0.record()
            for _ in range(5):
                plan.fbp_backproject(d, img)
            e1.record()
            torch.cuda.synchronize()
            best.append(e0.elapsed_time(e1))
        ms[k], imgs[k] = min(best), img
        plan.close()
    assert torch.equal(imgs[few][0], imgs[1][0]) and torch.equal(imgs[many][0], imgs[1][0])
    k = min(few, many)
    assert torch.equal(imgs[few][:k], imgs[many][:k])
    assert ms[many] <= limit * ms[few], ms
