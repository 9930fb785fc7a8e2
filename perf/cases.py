"""The performance cases of the CT-XAFS reconstruction library.

Each case is one call (or one short sequence of calls) that a reconstruction program makes on
device data through the package's public entry points: the OS-EM of one slice and of batches of
slices, CT-XAFS stacks of uneven slices through a batch plan, the differentiable projector pair,
filtered backprojection, the compressed-sensing OS-EM, the rotation-centre search, and the
reslicing of a projection stack.  ``listed()`` holds one case of each use at a size that it has
in earnest, from a 256 x 256 slice, where launches and latency count, to ten slices of
2048 x 2048; ``draw()`` gives more cases of the same ranges, odd sizes among them.

Inputs are made on the GPU from the seed alone: analytic sinograms of random ellipses with
transmission (Poisson) noise and a log conversion, as an experiment delivers them, without any
projector of this library.  ``exact()`` restates each result in 64 bits with torch operations:
the forward model's bilinear ray sums, the ratio, the backprojections and the updates are
evaluated in float64.  The choice of a detector bin by the nearest rule is part of the
reconstruction's definition (a rounded float32 expression, discontinuous in its arguments), so
the bins are those of that float32 expression; likewise the angle table is the float32
one that every plan uses, and the focus mask's comparisons.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ct-xafs_analysis_gb300"))

import xct  # noqa: E402
from xct import autograd as xag  # noqa: E402

DEV = "cuda"
INIT = 1.0  # the initial image of the iterative reconstructions (a constant image)
MAX_FLOPS = 9.0e11  # a drawn case costs no more than the largest listed one


# ------------------------------------------------------------------------------------ cases
def listed():
    return [
        # one 256^2 slice, 180 angles, 10 subsets x 5 iterations: the interactive preview of one
        # slice; 100+ dependent steps of a few microseconds of work
        dict(name="osem_256_one", op="osem", n=256, ny=256, px=256, pa=180, ss=10, it=5, slices=1, center=-1.0, cover=0),
        # the same, ten slices per call (the reference's default batch)
        dict(name="osem_256_ten", op="osem", n=256, ny=256, px=256, pa=180, ss=10, it=5, slices=10, center=-1.0, cover=0),
        # three slices of an odd, non-square size with an off-centre axis and a subset count that
        # does not divide the angles: a cropped scan as it comes
        dict(name="osem_509_odd", op="osem", n=509, ny=487, px=521, pa=367, ss=12, it=2, slices=3, center=257.25, cover=1),
        # one slice at full size: one iteration of 15 subsets over 1500 angles
        dict(name="osem_2048_one", op="osem", n=2048, ny=2048, px=2048, pa=1500, ss=15, it=1, slices=1, center=-1.0, cover=0),
        # the library's headline workload: ten full-size slices per call
        dict(name="osem_2048_ten", op="osem", n=2048, ny=2048, px=2048, pa=1500, ss=15, it=1, slices=10, center=-1.0, cover=0),
        # a CT-XAFS stack: slices of uneven widths and angle lists (an energy scan), two per
        # geometry, through one batch plan
        dict(name="stack_uneven", op="stack", widths="512,1024,1536,2048", angles="360,720,900,1200", geometries=12, each=2, shapes=3, ss=10, it=1),
        # the differentiable projector and its adjoint on one 1024^2 slice (a gradient step of a
        # model-based or learned reconstruction)
        dict(name="pair_1024_one", op="pair", n=1024, ny=1024, px=1024, pa=720, slices=1, center=-1.0),
        # the same for ten slices at once
        dict(name="pair_1024_ten", op="pair", n=1024, ny=1024, px=1024, pa=720, slices=10, center=-1.0),
        # filtered backprojection of one full-size slice
        dict(name="fbp_2048_one", op="fbp", n=2048, ny=2048, px=2048, pa=1500, zp=4096, slices=1, center=-1.0),
        # compressed-sensing OS-EM of ten half-size slices, coupled across slices
        dict(name="cs_512_ten", op="cs", n=512, ny=512, px=512, pa=360, ss=10, it=2, slices=10, center=-1.0, lam=1.0e-4),
        # the rotation-centre search that precedes every reconstruction: 16 candidate shifts
        dict(name="center_1024", op="center", n=1024, ny=1024, px=1024, pa=360, ss=10, shifts=16, start=-4.0, step=0.5),
        # reslicing a drift-corrected projection stack into sinograms, then the spike filter
        dict(name="reslice_2048", op="reslice", w=2048, h=48, a=720, corr=1, thr=0.05),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _limit(case, key):
    """The case with as many slices (shifts, geometries) as the largest listed case's cost allows."""
    case[key] = max(1, min(case[key], int(MAX_FLOPS / max(1.0, work({**case, key: 1})["flops"]))))
    return case


def draw(rng):
    op = rng.choice(["osem", "osem", "osem", "osem", "osem", "stack", "pair", "pair", "fbp", "cs", "center", "reslice"])
    n = _log_int(rng, 64, 2048)
    if rng.random() < 0.5:
        n = max(64, 32 * (n // 32))  # half of the sizes are round, half are as they fall
    ny = n if rng.random() < 0.6 else max(48, int(n * rng.uniform(0.7, 1.2)))
    ny = min(ny, 2048)
    px = n if rng.random() < 0.6 else max(48, int(n * rng.uniform(0.9, 1.3)))
    pa = max(24, int(n * rng.uniform(0.35, 1.0)))
    center = -1.0 if rng.random() < 0.5 else round(px * 0.5 + rng.uniform(-0.03, 0.03) * px, 2)
    ss = rng.choice([4, 6, 8, 10, 12, 15, 16])
    slices = rng.choice([1, 1, 2, 3, 5, 8, 10, 12, 16])
    if op == "osem":
        return _limit(dict(op=op, n=n, ny=ny, px=px, pa=pa, ss=ss, it=rng.choice([1, 2, 3, 5]) if n <= 1024 else 1,
                           slices=slices, center=center, cover=rng.choice([0, 0, 1])), "slices")
    if op == "stack":
        lo = _log_int(rng, 128, 1024)
        widths = sorted({lo, int(lo * 1.5), lo * 2, rng.randint(lo, 2 * lo)})
        angles = sorted({max(24, int(w * rng.uniform(0.4, 0.8))) for w in widths})
        return _limit(dict(op=op, widths=",".join(map(str, widths)), angles=",".join(map(str, angles)),
                           geometries=rng.randint(2, 12), each=rng.choice([1, 2, 3, 8]), shapes=rng.randint(1, 10 ** 6),
                           ss=rng.choice([6, 8, 10]), it=1), "geometries")
    if op == "pair":
        return _limit(dict(op=op, n=min(n, 1400), ny=min(ny, 1400), px=px, pa=min(pa, 900), slices=slices, center=center), "slices")
    if op == "fbp":
        zp = 64
        while zp < px * rng.choice([1, 2]):
            zp *= 2
        return _limit(dict(op=op, n=n, ny=ny, px=px, pa=pa, zp=zp, slices=slices, center=center), "slices")
    if op == "cs":
        n, ny = min(n, 1024), min(ny, 1024)
        return _limit(dict(op=op, n=n, ny=ny, px=min(px, 1300), pa=min(pa, 720), ss=ss, it=rng.choice([1, 2]), slices=max(2, slices),
                           center=center, lam=rng.choice([1.0e-4, 1.0e-3])), "slices")
    if op == "center":
        n = min(n, 1024)
        return _limit(dict(op=op, n=n, ny=n, px=n, pa=min(pa, 720), ss=ss, shifts=rng.choice([8, 11, 16, 21]),
                           start=-float(rng.randint(2, 6)), step=0.5), "shifts")
    return dict(op="reslice", w=_log_int(rng, 256, 2048), h=rng.randint(8, 64), a=rng.randint(90, 900), corr=rng.choice([0, 1]), thr=0.05)


# ----------------------------------------------------------------------------- what it takes
def _overlap(n, ny, px, pa):
    """Samples of the forward model that meet the image, and (pixel, angle) pairs that land on
    the detector, over pa angles of half a turn (the mean over angles of the area in which the
    image, a rectangle, meets the strip of the detector and the rays' length)."""
    th = np.linspace(0.0, math.pi, 64, endpoint=False)
    y, x = np.mgrid[0:32, 0:32]
    x, y = (x.ravel() + 0.5) / 32 * n - n / 2, (y.ravel() + 0.5) / 32 * ny - ny / 2
    c, s = np.cos(th)[:, None], np.sin(th)[:, None]
    on = np.abs(x * c - y * s) < px / 2
    in_ray = np.abs(x * s + y * c) < max(n, ny) / 2
    return float((on & in_ray).mean()) * n * ny * pa, float(on.mean()) * n * ny * pa


def _osem_flops(n, ny, px, pa, ss, it):
    # 12 operations for a bilinear sample and its sum, 5 for a nearest-bin gather, 4 for an update
    t_fwd, t_bp = _overlap(n, ny, px, pa)
    return it * (12 * t_fwd + 5 * t_bp + 4.0 * n * ny * ss)


def work(case):
    op = case["op"]
    if op == "reslice":
        px = case["w"] * case["h"] * case["a"]
        return {"bytes": 4.0 * px * 2 * 2, "flops": 30.0 * px}  # reslice and filter: each reads and writes the stack
    if op == "stack":
        items = _stack_items(case)
        return {"bytes": float(sum(4 * (w * len(a) + w * w) for w, a in items)),
                "flops": float(sum(_osem_flops(w, w, w, len(a), case["ss"], case["it"]) for w, a in items))}
    n, ny, px, pa = case["n"], case["ny"], case["px"], case["pa"]
    t_fwd, t_bp = _overlap(n, ny, px, pa)
    img, sino = 4.0 * n * ny, 4.0 * px * pa
    if op == "pair":  # image in, projection out; gradient in, image gradient out
        k = case["slices"]
        return {"bytes": k * 2 * (img + sino), "flops": k * 24.0 * t_fwd}
    if op == "fbp":  # two transforms of a padded row (5 zp log2 zp, two rows at once), a lerp and a sum per gather
        k = case["slices"]
        return {"bytes": k * (img + sino), "flops": k * (9.0 * t_bp + 5.0 * case["zp"] * math.log2(case["zp"]) * pa)}
    if op == "center":
        k = case["shifts"]
        return {"bytes": sino + k * img, "flops": k * (_osem_flops(n, ny, px, pa, case["ss"], 1) + 25.0 * n * ny)}
    k = case["slices"]
    flops = k * _osem_flops(n, ny, px, pa, case["ss"], case["it"])
    if op == "cs":  # the proximal step: a sort of six neighbours and 12 selections per voxel and subset
        flops += k * 60.0 * n * ny * case["ss"] * case["it"]
    return {"bytes": k * (img + sino), "flops": flops}


# ----------------------------------------------------------------------------------- inputs
def _angles(pa):
    return (np.arange(pa, dtype=np.float64) * (180.0 / pa)).astype(np.float32)


def _trig(angles):
    """(cos, sin) of every angle as the plans tabulate them: float32 radians, float32 results."""
    phi = (np.asarray(angles, np.float32).astype(np.float64) * math.pi / 180.0).astype(np.float32).astype(np.float64)
    return np.cos(phi).astype(np.float32), np.sin(phi).astype(np.float32)


def _stack_items(case):
    """(width, angle list) of every item of a stack: uneven widths and projection counts, some
    angles dropped, `each` consecutive slices per geometry."""
    rng = np.random.RandomState(case["shapes"])
    widths = [int(v) for v in case["widths"].split(",")]
    angles = [int(v) for v in case["angles"].split(",")]
    out = []
    for _ in range(case["geometries"]):
        w, pa = int(rng.choice(widths)), int(rng.choice(angles))
        drop = int(rng.randint(0, pa // 10 + 1))
        keep = np.sort(rng.permutation(pa)[: pa - drop])
        out += [(w, (keep * (180.0 / pa)).astype(np.float32))] * case["each"]
    return out


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _ellipses(rng, n, ny, count):
    """Rows (x, y, a, b, angle, density) of random ellipses in the inner field of view."""
    m = min(n, ny)
    r, t = 0.35 * m * np.sqrt(rng.uniform(0, 1, count)), rng.uniform(0, 2 * math.pi, count)
    a, b = rng.uniform(0.03, 0.25, count) * m, rng.uniform(0.03, 0.25, count) * m
    return np.stack([n / 2 + r * np.cos(t), ny / 2 + r * np.sin(t), a, b, rng.uniform(0, math.pi, count),
                     rng.uniform(0.2, 1.0, count) * 8.0 / m], axis=1)


def _sinogram(rng, gen, n, ny, px, angles, center, slices, i0=5.0e4):
    """Noisy log sinograms [slices][pa][px] of random ellipses (exact line integrals)."""
    cx = px * 0.5 if center < 0 else center
    th = torch.from_numpy(np.asarray(angles, np.float64) * math.pi / 180.0).to(DEV)[:, None]
    c, s = torch.cos(th), torch.sin(th)
    u = torch.arange(px, device=DEV, dtype=torch.float64)[None, :] - cx
    p = torch.zeros((slices, len(angles), px), device=DEV, dtype=torch.float64)
    base = _ellipses(rng, n, ny, 6)
    for z in range(slices):
        e = base.copy()  # neighbouring slices of one sample: the same bodies, slightly changed
        e[:, :2] += rng.uniform(-0.02, 0.02, (len(e), 2)) * min(n, ny)
        e[:, 5] *= rng.uniform(0.8, 1.2, len(e))
        for x0, y0, a, b, al, mu in e:
            t = u - ((x0 - n * 0.5) * c - (y0 - ny * 0.5) * s)
            # the ray normal (c, -s) in the ellipse's axes
            r2 = (a * (c * math.cos(al) - s * math.sin(al))) ** 2 + (b * (c * math.sin(al) + s * math.cos(al))) ** 2
            p[z] += (2.0 * a * b * mu) * torch.sqrt(torch.clamp(r2 - t * t, min=0.0)) / r2
    counts = torch.poisson(i0 * torch.exp(-p), generator=gen)
    return (-torch.log(torch.clamp(counts, min=1.0) / i0)).float()


def _image(rng, gen, n, ny, slices):
    """Images [slices][ny][nx]: ellipses and a smooth texture, as an iterate of a reconstruction."""
    y, x = torch.meshgrid(torch.arange(ny, device=DEV, dtype=torch.float32), torch.arange(n, device=DEV, dtype=torch.float32),
                          indexing="ij")
    img = torch.rand((slices, ny, n), device=DEV, generator=gen) * 0.002
    for z in range(slices):
        for x0, y0, a, b, al, mu in _ellipses(rng, n, ny, 6):
            ca, sa = math.cos(al), math.sin(al)
            d = (((x - x0) * ca + (y - y0) * sa) / a) ** 2 + (((y - y0) * ca - (x - x0) * sa) / b) ** 2
            img[z] += float(mu) * (d <= 1.0)
    return img


def _make(case, seed):
    """The inputs of a case, as a dict of tensors (what prepare() and exact() start from)."""
    rng, gen = np.random.RandomState((int(seed) * 7919 + 17) % (1 << 31)), _gen(seed)
    op = case["op"]
    if op == "reslice":
        w, h, a = case["w"], case["h"], case["a"]
        proj = torch.rand((a, h, w), device=DEV, generator=gen) * 0.02
        col = torch.linspace(0.0, math.pi, w, device=DEV)
        proj += (1.5 * torch.sin(col))[None, None, :] * torch.linspace(0.6, 1.0, h, device=DEV)[None, :, None]
        proj[torch.rand((a, h, w), device=DEV, generator=gen) < 0.001] += 0.3  # one-angle spikes (zingers)
        return {"proj": proj, "xs": rng.uniform(-2, 2, a).astype(np.float32), "ys": rng.uniform(-1.5, 1.5, a).astype(np.float32)}
    if op == "stack":
        return {"sinos": [_sinogram(rng, gen, w, w, w, ang, -1.0, 1)[0].contiguous() for w, ang in _stack_items(case)]}
    ang = _angles(case["pa"])
    if op == "pair":
        return {"x": _image(rng, gen, case["n"], case["ny"], case["slices"]),
                # the gradient of a data term: a projection-like residual of both signs
                "g": torch.randn((case["slices"], case["pa"], case["px"]), device=DEV, generator=gen)}
    if op == "center":
        return {"sino": _sinogram(rng, gen, case["n"], case["ny"], case["px"], ang, case["px"] * 0.5 + 1.0, 1)}
    return {"sino": _sinogram(rng, gen, case["n"], case["ny"], case["px"], ang, case["center"], case["slices"])}


def prepare(case, seed):
    st = {"case": dict(case), **_make(case, seed)}
    op = case["op"]
    ctx = st["ctx"] = xct.Context(0)
    if op == "reslice":
        st["plan"] = xct.ReslicePlan(ctx, case["w"], case["h"], case["a"], st["xs"], st["ys"], 0.0, case["corr"])
        st["out"] = torch.empty((case["h"], case["a"], case["w"]), device=DEV)
        st["den"] = torch.empty_like(st["out"])
    elif op == "stack":
        items = _stack_items(case)
        st["plan"] = xct.BatchPlan(ctx, [xct.make_geom(w, w, w, a, case["ss"], case["it"]) for w, a in items], case["it"])
        st["sizes"] = [w for w, _ in items]
    else:
        center = case.get("center", -1.0)
        st["plan"] = xct.OSEMPlan(ctx, case["n"], case["ny"], case["px"], _angles(case["pa"]), case.get("ss", 1), case.get("it", 1),
                                  center_bin=None if center < 0 else center,
                                  subset_mode=xct.SUBSETS_COVER if case.get("cover") else xct.SUBSETS_REF,
                                  max_batch=case["slices"] if "slices" in case else case["shifts"])
        if op == "pair":
            st["x"].requires_grad_(True)
    return st


def run(st):
    case, plan = st["case"], st["plan"]
    op = case["op"]
    if op == "reslice":
        plan.reslice(st["proj"], st["out"])
        xct.denoise_sinogram(st["out"], st["den"], case["thr"])
        return [st["out"], st["den"]]
    if op == "stack":
        pool = torch.full((sum(w * w for w in st["sizes"]),), INIT, device=DEV)
        imgs, at = [], 0
        for w in st["sizes"]:
            imgs.append(pool[at:at + w * w].view(w, w))
            at += w * w
        plan.run(st["sinos"], imgs)
        return imgs
    if op == "pair":
        y = xag.project(st["x"], plan)
        (gx,) = torch.autograd.grad(y, st["x"], st["g"])
        return [y.detach(), gx]
    if op == "fbp":
        img = torch.empty((case["slices"], case["ny"], case["n"]), device=DEV)
        plan.fbp(st["sino"], img, zp=case["zp"])
        return img
    if op == "center":
        imgs = torch.empty((case["shifts"], case["ny"], case["n"]), device=DEV)
        fi, best = plan.rot_center_search(st["sino"], imgs, case["start"], case["step"], init_value=INIT)
        return [imgs, fi, best]
    img = torch.full((case["slices"], case["ny"], case["n"]), INIT, device=DEV)
    if op == "cs":
        plan.cs_run_device(st["sino"], img, cs_lambda=case["lam"])
    else:
        plan.run_device(st["sino"], img)
    return img


# --------------------------------------------------------------------------------- 64 bits
class _Geom:
    """One geometry in float64: the sample positions of the forward model and the bins."""

    def __init__(self, n, ny, px, angles, center):
        self.n, self.ny, self.px, self.pa = n, ny, px, len(angles)
        self.cx = px * 0.5 if center < 0 else float(np.float32(center))
        self.d = max(n, ny)
        self.c32, self.s32 = _trig(angles)
        self.c, self.s = self.c32.astype(np.float64), self.s32.astype(np.float64)
        f = dict(device=DEV, dtype=torch.float64)
        self.xr = torch.arange(px, **f)[:, None] - self.cx
        self.yr = torch.arange(self.d, **f)[None, :] - self.d * 0.5

    def taps(self, th):
        """The four footprint cells in the zero-bordered image and the weights of every sample."""
        c, s = float(self.c[th]), float(self.s[th])
        x = self.yr * s + self.xr * c + self.n * 0.5
        y = self.yr * c - self.xr * s + self.ny * 0.5
        fi, fj = torch.floor(x), torch.floor(y)
        a, b = x - fi, y - fj
        i, j = fi.to(torch.int64), fj.to(torch.int64)
        i0, i1 = (i + 1).clamp_(0, self.n + 1), (i + 2).clamp_(0, self.n + 1)
        j0, j1 = (j + 1).clamp_(0, self.ny + 1) * (self.n + 2), (j + 2).clamp_(0, self.ny + 1) * (self.n + 2)
        for cell, w in ((j0 + i0, (1 - a) * (1 - b)), (j0 + i1, a * (1 - b)), (j1 + i0, (1 - a) * b), (j1 + i1, a * b)):
            yield cell.view(-1), w.view(-1)

    def pad(self, img):
        """Images [k][ny][nx] as [(ny + 2)(nx + 2)][k] with a border of zeros."""
        p = torch.zeros((self.ny + 2, self.n + 2, img.shape[0]), device=DEV, dtype=torch.float64)
        p[1:-1, 1:-1] = img.permute(1, 2, 0)
        return p.view(-1, img.shape[0])

    def forward(self, pad, th):
        """Ray sums [px][k] of angle th."""
        acc = 0.0
        for cell, w in self.taps(th):
            acc = acc + w[:, None] * pad[cell]
        return acc.view(self.px, self.d, -1).sum(1)

    def bins32(self, th):
        """The nearest detector bin of every pixel: ((Xc c - Yc s) + cx) + 0.5 in float32."""
        f = dict(device=DEV, dtype=torch.float32)
        xc = torch.arange(self.n, **f)[None, :] - self.n * 0.5
        yc = torch.arange(self.ny, **f)[:, None] - self.ny * 0.5
        c, s = torch.tensor(self.c32[th], **f), torch.tensor(self.s32[th], **f)
        t = ((xc * c - yc * s) + self.cx) + 0.5
        return torch.floor(t).to(torch.int64)

    def bin_lookup(self, row, bins):
        """row [k][px] at integer bins, zero off the detector -> [k][ny][nx]."""
        p = torch.zeros((row.shape[0], self.px + 2), device=DEV, dtype=torch.float64)
        p[:, 1:-1] = row
        return p[:, (bins + 1).clamp(0, self.px + 1)]


def _subset_order(ss):
    if ss & (ss - 1):
        return list(range(ss))
    bits = ss.bit_length() - 1
    return [int(format(k, "0%db" % bits)[::-1], 2) if bits else 0 for k in range(ss)]


def _osem_step64(g, meas, img, ratio, ss, sub, cover):
    """One OS-EM subset step on images [k][ny][nx] from sinograms meas [k][pa][px], in float64."""
    rows = (g.pa - sub + ss - 1) // ss if cover else g.pa // ss
    pad = g.pad(img)
    for th in range(sub, sub + rows * ss, ss):
        p = g.forward(pad, th).t()
        m = torch.where(meas[:, th] > 1.0e-6, meas[:, th], torch.full_like(p, 1.0e-6))
        ratio[:, th] = torch.where(p < 1.0e-4, m, m / p)
    b = torch.zeros_like(img)
    for th in range(sub, g.pa, ss):
        b += g.bin_lookup(ratio[:, th], g.bins32(th))
    return img * b * ss / g.pa


def _osem64(g, sino, ss, it, cover=0):
    meas = sino.double()
    img = torch.full((sino.shape[0], g.ny, g.n), INIT, device=DEV, dtype=torch.float64)
    ratio = torch.zeros_like(meas)
    for _ in range(it):
        for sub in _subset_order(ss):
            img = _osem_step64(g, meas, img, ratio, ss, sub, cover)
    return img


def _prox64(v, lam, floor):
    """The six-neighbour proximal step on images [k][ny][nx]: x +- 1 and y +- 1 with a zero
    border, the next slice (the last one's own), and the first slice."""
    k = v.shape[0]
    p = torch.nn.functional.pad(v, (1, 1, 1, 1))
    nb = torch.stack([p[:, 1:-1, 2:], p[:, 1:-1, :-2], p[:, 2:, 1:-1], p[:, :-2, 1:-1],
                      v[[min(z + 1, k - 1) for z in range(k)]], v[0:1].expand_as(v)])
    nb = torch.sort(nb, dim=0, descending=True).values
    l2, l4, l6 = 2 * lam, 4 * lam, 6 * lam
    cand = [v - l6, nb[0], v - l4, nb[1], v - l2, nb[2], v, nb[3], v + l2, nb[4], v + l4, nb[5], v + l6]
    edge = [nb[0] + l6, nb[0] + l4, nb[1] + l4, nb[1] + l2, nb[2] + l2, nb[2], nb[3], nb[3] - l2, nb[4] - l2, nb[4] - l4,
            nb[5] - l4, nb[5] - l6]
    x = cand[0]
    for e, c in zip(edge, cand[1:]):
        x = torch.where(v < e, c, x)
    return x.clamp(min=1.0e-6) if floor else x


def _cs64(g, sino, ss, it, lam):
    meas = sino.double()
    img = torch.full((sino.shape[0], g.ny, g.n), INIT, device=DEV, dtype=torch.float64)
    ratio = torch.zeros_like(meas)
    lam = float(np.float32(float("%g" % np.float32(lam))))
    first = True
    for _ in range(it):
        for sub in _subset_order(ss):
            # the first step's proximal operator takes the image before its OS-EM update
            img = _prox64(img, lam, True) if first else _prox64(_osem_step64(g, meas, img, ratio, ss, sub, 0), lam, False)
            first = False
    return img


def _fbp64(g, sino, zp):
    k = sino.shape[0]
    ramp = torch.arange(zp, device=DEV, dtype=torch.float64)
    ramp = torch.minimum(ramp, zp - ramp) * (math.pi / zp)
    img = torch.zeros((k, g.ny, g.n), device=DEV, dtype=torch.float64)
    f = dict(device=DEV, dtype=torch.float64)
    xc = torch.arange(g.n, **f)[None, :] - g.n * 0.5
    yc = torch.arange(g.ny, **f)[:, None] - g.ny * 0.5
    filt = torch.fft.ifft(torch.fft.fft(sino.double(), n=zp, dim=2) * ramp, dim=2).real[:, :, :g.px]
    for th in range(g.pa):
        u = xc * float(g.c[th]) - yc * float(g.s[th]) + g.cx
        i = torch.floor(u)
        a, i = u - i, i.to(torch.int64)
        img += (1 - a) * g.bin_lookup(filt[:, th], i) + a * g.bin_lookup(filt[:, th], i + 1)
    return img / (2.0 * g.pa) * (torch.sqrt(xc * xc + yc * yc) < g.n * 0.5)


def _mask32(g, shift, a0, a1):
    """The focus index's mask of one shift, [ny][nx] (float32 comparisons)."""
    f32 = np.float32
    half = f32(g.n // 2)
    rp, rm = min(half + f32(shift), half), max(-half + f32(shift), -half)

    def axes(ang):
        return (f32(math.cos(float(f32(float(f32(ang)) * math.pi / 180)))),
                f32(math.cos(float(f32(float(f32(ang)) * math.pi / 180 - math.pi / 2)))))
    lo, hi = axes(a0), axes(a1)
    t = lambda v: torch.tensor(f32(v), device=DEV, dtype=torch.float32)  # noqa: E731
    x = torch.arange(g.n, device=DEV, dtype=torch.float32)[None, :] - t(half)
    y = torch.arange(g.ny, device=DEV, dtype=torch.float32)[:, None] - t(g.ny // 2)
    rp2, rm2 = f32(rp * rp), f32(rm * rm)
    dot = lambda r, ax: x * t(f32(r * ax[0])) + y * t(f32(r * ax[1]))  # noqa: E731
    m = (dot(rp, hi) <= t(rp2)) & (dot(rp, lo) <= t(rp2)) & (dot(rm, hi) <= t(rm2)) & (dot(rm, lo) <= t(rm2))
    pd = t(f32((rp if rp2 < rm2 else rm) * hi[0]))
    d2 = x * x + y * y
    return m & (((d2 <= t(rp2)) & (x > pd)) | ((d2 <= t(rm2)) & (x <= pd)))


def _focus64(g, img, mask):
    m = torch.zeros((g.ny + 2, g.n + 2), device=DEV, dtype=torch.bool)
    m[1:-1, 1:-1] = mask
    p = torch.nn.functional.pad(img, (1, 1, 1, 1))
    ok, sq = mask.clone(), torch.zeros_like(img)
    for dy in (0, 1, 2):
        for dx in (0, 1, 2):
            ok &= m[dy:dy + g.ny, dx:dx + g.n]
            sq += (p[dy:dy + g.ny, dx:dx + g.n] - img) ** 2
    return float(torch.sqrt((sq / img ** 2)[ok].sum() / ok.sum()))


def _reslice64(case, d):
    w, h, a = case["w"], case["h"], case["a"]
    proj = torch.nn.functional.pad(d["proj"].double(), (1, 1, 1, 1))
    out = torch.empty((h, a, w), device=DEV, dtype=torch.float64)
    f = dict(device=DEV, dtype=torch.float64)
    x, y = torch.arange(w, **f), torch.arange(h, **f)
    fac = torch.sqrt(torch.clamp(1.0 - (2.0 * (x - w * 0.5).abs() / w) ** 2, min=0.0)) if case["corr"] else 1.0
    for th in range(a):
        u, v = x + float(d["xs"][th]), y + float(d["ys"][th])
        i, j = torch.floor(u), torch.floor(v)
        p, q = u - i, (v - j)[:, None]
        i, j = i.to(torch.int64), j.to(torch.int64)
        at = lambda di, dj: proj[th][(j + 1 + dj).clamp(0, h + 1)][:, (i + 1 + di).clamp(0, w + 1)]  # noqa: E731
        out[:, th] = ((1 - q) * ((1 - p) * at(0, 0) + p * at(1, 0)) + q * ((1 - p) * at(0, 1) + p * at(1, 1))) * fac
    before, after = torch.cat([out[:, :1], out[:, :-1]], 1), torch.cat([out[:, 1:], out[:, -1:]], 1)
    d1, d2, t = after - out, out - before, case["thr"]
    spike = ((d1 > t) & (d2 < -t)) | ((d1 < -t) & (d2 > t))
    return [out, torch.where(spike, (after + before) * 0.5, out)]


def exact(case, seed):
    d = _make(case, seed)
    op = case["op"]
    if op == "reslice":
        return _reslice64(case, d)
    if op == "stack":
        return [_osem64(_Geom(w, w, w, a, -1.0), s[None], case["ss"], case["it"])[0] for (w, a), s in zip(_stack_items(case), d["sinos"])]
    g = _Geom(case["n"], case["ny"], case["px"], _angles(case["pa"]), case.get("center", -1.0))
    if op == "pair":
        k = case["slices"]
        x, gr = g.pad(d["x"].double()), d["g"].double()
        y = torch.empty((k, g.pa, g.px), device=DEV, dtype=torch.float64)
        back = torch.zeros_like(x)
        for th in range(g.pa):
            y[:, th] = g.forward(x, th).t()
            rays = gr[:, th].t().repeat_interleave(g.d, dim=0)
            for cell, w in g.taps(th):
                back.index_add_(0, cell, w[:, None] * rays)
        return [y, back.view(g.ny + 2, g.n + 2, k)[1:-1, 1:-1].permute(2, 0, 1).contiguous()]
    if op == "fbp":
        return _fbp64(g, d["sino"], case["zp"])
    if op == "cs":
        return _cs64(g, d["sino"], case["ss"], case["it"], case["lam"])
    if op == "center":
        s = d["sino"][0].double()
        p = torch.nn.functional.pad(s, (1, 1))
        x = torch.arange(g.px, device=DEV, dtype=torch.float64)
        shifted = []
        for i in range(case["shifts"]):
            u = x + (case["start"] + case["step"] * i)
            fi = torch.floor(u)
            a, b = u - fi, fi.to(torch.int64)
            shifted.append((1 - a) * p[:, (b + 1).clamp(0, g.px + 1)] + a * p[:, (b + 2).clamp(0, g.px + 1)])
        img = _osem64(g, torch.stack(shifted), case["ss"], 1)
        ang = _angles(case["pa"])
        fi = [_focus64(g, img[i], _mask32(g, case["start"] + case["step"] * i, ang[0], ang[-1])) for i in range(case["shifts"])]
        return [img, np.array(fi), None]
    return _osem64(g, d["sino"], case["ss"], case["it"], case["cover"])
