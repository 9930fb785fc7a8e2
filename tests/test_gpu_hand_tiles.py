"""A forward tile set by hand is the forward projector's choice and nothing else's.  On a ten-slice plan large
enough for the slice-interleaved kernels, after set_tuning: whole groups of eight stay in the grouped
forward form and the two slices left take the tile (two launches and the ratio's); the backprojection stays
in a group of eight and a pair; the adjoint of eight slices stays the gather, whose float sums have a fixed
order, so its image is the same bits (the two others are scattered together).  The ray sums agree to the bar of the forms against each other, 1e-6 rel-L2."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def test_hand_tile_leaves_the_other_kernels_grouped(gpu_ctx):
    import xct
    n, pa, ss, dN = 740, 14, 2, 10
    ang = (np.arange(pa) * (180.0 / pa)).astype(np.float32)
    plan = xct.OSEMPlan(gpu_ctx, n, n, n, ang, ss, 1, max_batch=dN)
    assert plan.multislice() == 128
    gen = torch.Generator().manual_seed(3)
    img = (torch.rand((dN, n, n), generator=gen) + 0.1).cuda()
    y = torch.randn((dN, pa, n), generator=gen).cuda()

    def run():
        out, counts = [], []
        for call in ("fwd", "adj", "osem2"):
            o = img.clone() if call == "osem2" else torch.empty_like(y if call == "fwd" else img)
            n0 = xct.launch_count()
            if call == "fwd":
                plan.fwd(img, o)
            elif call == "adj":
                plan.adj(y, o)
            else:
                plan.osem2(1, o, y.abs())
            counts.append(xct.launch_count() - n0)
            out.append(o.cpu().numpy())
        return out, counts

    before, n_before = run()
    plan.set_tuning(60, 16)
    assert plan.tuning() == (60, 16) and plan.multislice() == 128
    after, n_after = run()
    fwd_launches = -(-pa // (pa // ss))  # the accumulator holds a subset's rows
    assert n_before == [3 * fwd_launches, 2, 2]
    assert n_after == [3 * fwd_launches, 2, 2]
    a, b = before[0].astype(np.float64), after[0].astype(np.float64)
    assert np.linalg.norm(a - b) <= 1e-6 * np.linalg.norm(b)
    assert np.array_equal(before[1][:8], after[1][:8])
    assert np.array_equal(before[2], after[2])
    plan.close()
