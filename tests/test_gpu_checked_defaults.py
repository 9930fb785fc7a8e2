"""The bounds-checked build over the kernels that plans take by themselves (tests/test_gpu_checked.py runs them
with tiles by hand): the forward tiles of one to five slices, large and small, in runs and in the batch graph's
packs and large single slices, the one-, two-, four- and eight-slice backprojectors, the FBP ones, and the
adjoint's scatter tiles and gather groups, at awkward sizes.  No access may fall outside its buffer, and the
results equal the standard library's."""
import os
import subprocess
import sys

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "ct-xafs_analysis_gb300")

RUN = r"""
import sys, numpy as np, torch, xct
PLANS = [  # nx, ny, px, angles, span, centre offset, slices
    (501, 470, 520, 40, 180.0, 3.25, 1), (330, 301, 290, 36, 360.0, -7.5, 2), (163, 400, 500, 31, 180.0, 0.0, 3),
    (301, 277, 310, 30, 200.0, 11.25, 4), (260, 250, 300, 24, 180.0, 0.0, 5), (401, 390, 360, 20, 180.0, -2.0, 10),
    (760, 741, 770, 8, 180.0, 1.5, 13), (60, 77, 90, 20, 360.0, 4.0, 8), (1200, 1100, 1300, 6, 180.0, 0.0, 1)]
STACKS = [[(330, 320, 341, 42, 2.0, 7), (290, 300, 280, 40, 0.0, 3)], [(1000, 990, 1010, 260, -3.0, 1), (700, 800, 810, 200, 0.0, 1)]]
ctx = xct.Context(0)
out = {}
gen = torch.Generator().manual_seed(1)
rand = lambda *s: (torch.rand(s, generator=gen) + 0.2).cuda()
for i, (nx, ny, px, pa, span, off, dN) in enumerate(PLANS):
    ang = (np.arange(pa) * (span / pa)).astype(np.float32)
    plan = xct.OSEMPlan(ctx, nx, ny, px, ang, 2, 1, center_bin=px * 0.5 + off, max_batch=dN)
    img, y = rand(dN, ny, nx), rand(dN, pa, px)
    f, a, b, x = torch.empty_like(y), torch.empty_like(img), torch.empty_like(img), torch.ones_like(img)
    plan.fwd(img, f)
    plan.run_device(y, x)
    plan.adj(y, a)
    plan.fbp_backproject(y, b)
    torch.cuda.synchronize()
    for n, t in (("fwd", f), ("osem", x), ("adj", a), ("fbp", b)):
        out["%s_%d" % (n, i)] = t.cpu().numpy()
    plan.close()
for i, items in enumerate(STACKS):
    geoms, sinos, imgs = [], [], []
    for nx, ny, px, pa, off, count in items:
        for _ in range(count):
            geoms.append(xct.make_geom(nx, ny, px, (np.arange(pa) * (180.0 / pa)).astype(np.float32), 2, 1, center_bin=px * 0.5 + off))
            sinos.append(rand(pa, px))
            imgs.append(torch.ones((ny, nx), device="cuda"))
    bp = xct.BatchPlan(ctx, geoms, 1)
    bp.run(sinos, imgs)
    torch.cuda.synchronize()
    for k, t in enumerate(imgs):
        out["stack_%d_%d" % (i, k)] = t.cpu().numpy()
    bp.close()
np.savez(sys.argv[1], **out)
if len(sys.argv) > 2:
    print("CHECK", *xct.check_report(ctx))
"""


def test_default_kernels_stay_inside_their_buffers(xct_lib, tmp_path):
    sys.path.insert(0, PKG)
    from xct import build
    build.build_lib(checked=True)
    res = {}
    for variant in ("checked", ""):
        env = dict(os.environ, PYTHONPATH=PKG + os.pathsep + os.environ.get("PYTHONPATH", ""), XCT_LIB_VARIANT=variant)
        f = tmp_path / (variant + "r.npz")
        r = subprocess.run([sys.executable, "-c", RUN, str(f)] + (["report"] if variant else []), env=env,
                           capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
        if variant:
            line = [l for l in r.stdout.splitlines() if l.startswith("CHECK")][-1].split()
            assert int(line[1]) == 0, "skipped accesses: %s (site, index, lo, hi)" % line[1:]
        res[variant] = dict(np.load(f))
    a, b = res["checked"], res[""]
    assert set(a) == set(b)
    for k in a:
        if k.startswith("fbp"):  # the same sums in the same order
            assert np.array_equal(a[k], b[k]), k
        else:
            d = np.linalg.norm(a[k].astype(np.float64) - b[k])
            assert d <= 1e-6 * np.linalg.norm(b[k]), k
