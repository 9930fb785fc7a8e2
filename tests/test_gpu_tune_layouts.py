"""The batch autotuner's choice is for the slices that the graph serves one by one, and for no others.  A
stack of pairs is all packs: there is nothing to time, so nothing is stored (an untimed entry would answer for
the same shapes laid out as single slices).  With the grouping off the same plan has four single slices: the
autotuner times them (an entry with a time above zero), and a second plan of the same shapes with four
geometries -- no packs -- finds that entry.  Turned on again, the plan is back on its packs' tiles.  Every
layout gives the same images to the batch plan's bar, 1e-6 rel-L2."""
import json

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def test_choice_belongs_to_the_single_slices(gpu_ctx, tmp_path):
    import xct
    cache = tmp_path / "tune.json"
    shapes = [(301, 91), (337, 83)]  # sizes no other test tunes: the process keeps its choices too

    def entries():
        return json.loads(cache.read_text())["entries"] if cache.exists() else {}

    def plan(step):
        geoms = []
        for n, pa in shapes:
            for k in range(2):
                ang = ((np.arange(pa) + step * k) * (180.0 / pa)).astype(np.float32)
                geoms.append(xct.make_geom(n, n, n, ang, 4, 1))
        return xct.BatchPlan(gpu_ctx, geoms, 1)

    sinos = [torch.rand((pa, n), generator=torch.Generator().manual_seed(n)).cuda() + 0.5 for n, pa in shapes for _ in range(2)]

    def run(bp):
        imgs = [torch.ones((n, n), device="cuda") for n, _ in shapes for _ in range(2)]
        n0 = xct.launch_count()
        bp.run(sinos, imgs)
        torch.cuda.synchronize()
        return [x.cpu().numpy().astype(np.float64) for x in imgs], xct.launch_count() - n0

    bp = plan(0.0)
    first, launches = run(bp)
    assert launches == 3 * 4  # packs of two only
    bp.autotune(cache_path=cache)
    assert not entries()
    results = [run(bp)[0]]
    bp.set_grouping(False)
    results.append(run(bp)[0])
    bp.autotune(cache_path=cache)
    (key, entry), = entries().items()
    assert entry["ms"] > 0
    results.append(run(bp)[0])
    tile = bp.tuning()
    bp.set_grouping(True)
    results.append(run(bp)[0])
    bp.set_grouping(False)
    results.append(run(bp)[0])
    assert bp.tuning() == tile == (entry["fwd_tile"], entry["ang_chunk"])
    bp.close()
    for imgs in results:
        for a, b in zip(imgs, first):
            assert np.linalg.norm(a - b) <= 1e-6 * np.linalg.norm(b)
    other = plan(0.25)  # the second of each pair has its own angles
    assert other.autotune(cache_path=cache) == tile
    assert entries() == {key: entry}
    other.close()
