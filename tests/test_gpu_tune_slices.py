"""xct_plan_autotune times the launches that its choice serves.  With the grouping on, slices together go through
the grouped forms and the tuned tiles serve one slice, so eight slices' entry records the time of one
(within a factor of two of the entry tuned for one slice, a launch's noise included; 5 to 8 times it where
eight slices are timed).  With the grouping off the per-slice kernel serves all eight, and the entry is theirs."""
import json

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def test_autotune_times_what_it_chooses_for(gpu_ctx, tmp_path):
    import xct
    n, pa = 1023, 260  # a size no other test tunes
    ang = (np.arange(pa) * (180.0 / pa)).astype(np.float32)
    ms = {}
    for name, dN, off in (("one", 1, False), ("eight", 8, False), ("off", 8, True)):
        cache = tmp_path / (name + ".json")
        plan = xct.OSEMPlan(gpu_ctx, n, n, n, ang, 4, 1, max_batch=dN)
        if off:
            plan.set_multislice(0)
        plan.autotune(dN=dN, cache_path=cache, force=True)
        (key, e), = [(k, v) for k, v in json.loads(cache.read_text())["entries"].items() if "|%dx%d|" % (n, n) in k and "dN%d" % dN in k]
        ms[name] = e["ms"]
        plan.close()
    assert ms["eight"] <= 2.0 * ms["one"], ms
    assert ms["off"] >= 3.0 * ms["one"], ms
