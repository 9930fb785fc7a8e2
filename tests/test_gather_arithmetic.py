"""The gather adjoint's search as its kernel evaluates it (adj_gather_kernel in csrc/xct_adj.cu), in the
kernel's float32 operations (fused multiply-adds emulated exactly: float32 products are exact in float64), on the
CPU.  Per base texel (i, j) and angle the floors of (u, w) = di (c, s) + (dj (-s, c) + (cx, hd) - 0.717), plus
one, give the candidates Xa, Xa + 1 and Ya, Ya + 1; a candidate is kept when its offset from (i, j) is, as
bits, below those of 1.0 in x and in y (a negative offset has the sign bit).  In blocks that hold base texels -1
a negative coordinate is moved to at most -2^-24 first, whose offset from -1 is below 1.

Every forward sample must be among the candidates of its base texel and kept there, and kept by none of the
eight texels around it.  Sizes: odd and even, non-square, off-centre axes, detectors wider than the image up
to the largest (65536 bins, where a bin coordinate's spacing is 2^-8), the largest image side."""
import numpy as np
import pytest

f32 = np.float32

CASES = [  # nx, ny, px, cx
    (128, 128, 128, 64.0),
    (129, 97, 140, 73.25),
    (1, 3, 5, 2.5),
    (1023, 700, 1500, 741.3),
    (2048, 2048, 2048, 1024.0),
    (16383, 90, 16384, 8192.0),
    (300, 301, 65536, 65500.0),
    (512, 511, 65536, 65736.0),
]


def _fma(a, b, c):
    return (np.asarray(a, np.float64) * np.asarray(b, np.float64) + np.asarray(c, np.float64)).astype(f32)


@pytest.mark.parametrize("case", CASES)
def test_every_sample_is_kept_by_its_base_texel_alone(case):
    nx, ny, px, cx = case
    rng = np.random.default_rng(nx + ny)
    D = max(nx, ny)
    hx, hy, hd, cx = f32(nx * 0.5), f32(ny * 0.5), f32(D * 0.5), f32(cx)
    reach = np.hypot(nx, ny) / 2 + 2
    lo, hi = max(0, int(cx - reach)), min(px - 1, int(cx + reach))
    for deg in np.concatenate([[0.0, 45.0, 90.0, 135.0, 180.0, 270.0], rng.uniform(0.0, 360.0, 18)]):
        phi = np.float64(f32(np.float64(f32(deg)) * np.pi / 180.0))
        c, s = f32(np.cos(phi)), f32(np.sin(phi))
        X = np.unique(rng.integers(lo, hi + 1, 80))
        XX, YY = np.meshgrid(X, np.arange(D), indexing="ij")
        Xc, Yc = (XX.astype(f32) - cx).astype(f32), (YY.astype(f32) - hd).astype(f32)
        x, y = _fma(Yc, s, _fma(Xc, c, hx)), _fma(Yc, c, _fma(Xc, -s, hy))  # the forward's sample
        bi, bj = np.floor(x).astype(np.int64), np.floor(y).astype(np.int64)
        m = (bi >= -1) & (bi < nx) & (bj >= -1) & (bj < ny)
        bi, bj, sx, sy, x, y = bi[m], bj[m], XX[m], YY[m], x[m], y[m]
        for di_, dj_ in [(a, b) for a in (-1, 0, 1) for b in (-1, 0, 1)]:
            i, j = bi + di_, bj + dj_  # a texel that may look for this sample
            there = (i >= -1) & (i < nx) & (j >= -1) & (j < ny)
            fi, fj = i.astype(f32), j.astype(f32)
            di, dj = ((fi + f32(0.5)) - hx).astype(f32), ((fj + f32(0.5)) - hy).astype(f32)
            u = _fma(di, c, _fma(dj, -s, f32(cx - f32(0.717))))
            w = _fma(di, s, _fma(dj, c, f32(hd - f32(0.717))))
            Xa, Ya = np.floor(u).astype(np.int64) + 1, np.floor(w).astype(np.int64) + 1
            seen = ((sx == Xa) | (sx == Xa + 1)) & ((sy == Ya) | (sy == Ya + 1))
            for border in (False, True):  # blocks with and without base texels -1 (only the former hold them)
                gx, gy = x, y
                if border:
                    gx = np.where(x < 0, np.minimum(x, f32(-2.0 ** -24)), x)
                    gy = np.where(y < 0, np.minimum(y, f32(-2.0 ** -24)), y)
                ox, oy = (gx - fi).astype(f32).view(np.uint32), (gy - fj).astype(f32).view(np.uint32)
                kept = seen & (np.maximum(ox, oy) < 0x3F800000) & there
                where = there if border else there & (i >= 0) & (j >= 0)
                want = where if di_ == 0 and dj_ == 0 else np.zeros_like(where)
                assert np.array_equal(kept & where, want), (deg, di_, dj_, border)
