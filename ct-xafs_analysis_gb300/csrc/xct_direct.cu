// xct_direct.cu -- the OS-EM kernels for small problems.
//
// The tiled kernels (xct_tiled.cu) need hundreds of image tiles to fill 152 SMs; a 256 x 256
// slice has 36 forward tiles and 16 backprojection tiles.  Here the parallelism comes from the
// rays and from the pixels instead, and the image (or the ratio rows) is read through L1:
//   * fwd_direct_kernel: a CTA owns eight adjacent rays of one angle and splits their samples
//     over all its warps; it ends with the complete ray sums, so the OSEM1 ratio is formed in
//     the same launch (no accumulator, no atomics, no finalize launch);
//   * bp_direct_kernel: a thread owns one pixel of up to two slices and gathers its bins, in angle
//     order with the literal bin expression, so the image is the tiled kernel's bit for bit.
// Both are bound by latency at these sizes: a 256 x 256 slice with 18 angles per subset is 1.2 M
// samples, 8 per lane with every SM filled.  A subset step of it takes 10.4 us (the two launches
// overlap by programmatic stream serialization); 12.0 with the tiled forward kernel and its finalize (below).
#include "xct_device.cuh"
#include "xct_launch.cuh"
#include "xct_ray.cuh"

namespace {

constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
constexpr int kDirRays = 8, kDirLanes = 4;  // a warp reads 8 rays x 4 consecutive samples, a compact patch
constexpr int kDirWarps = 8;                // warps sharing the samples of the CTA's rays

// Where the small-problem kernels run.  They read texels through L1 at about 0.3 samples per ns
// whatever the size, the tiled forward kernels about 0.95 once their tiles fill the SMs; measured per
// subset step with both (taps in millions): 64^2 x 9 angles, one slice (0.04) 5.9 against 8.7 us; 128^2
// x 9 x ten slices (1.5) 13.6 against 17.0; 256^2 x 18, one (1.2) 10.8 against 12.0, three (3.5) 23.4
// against 17.8; 300^2 x 25, one (2.2) 16.4 against 13.9; 384^2 x 27, one (4.0) 25.2 against 17.9.  The
// line is drawn between 1.5 and 2.2.  The backprojector: one slice of 512^2 x 36 angles 4 against
// 14 us a launch, 1024^2 x 72 angles 46 against 31.
constexpr long long kDirectTaps = 1600000;  // image texels x subset angles x slices
constexpr long long kDirectPixels = 600000; // image pixels x slices

// grid: (ceil(px / 8), nrows, dN), kDirWarps warps.  meas != nullptr: OSEM1 ratio; else raw ray sums.
__global__ void __launch_bounds__(kDirWarps * 32) fwd_direct_kernel(const float *img, const float *meas, float *out,
                                                            const float2 *__restrict__ trig,
                                                            KGeom g, int sub, int step)
{
    constexpr int W = kDirWarps;
    __shared__ float part[W][kDirRays];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ray = lane / kDirLanes, ph = lane % kDirLanes;
    const int X = (int)blockIdx.x * kDirRays + ray;
    const int th = sub + (int)blockIdx.y * step, z = blockIdx.z;
    const float2 cs = __ldg(trig + th);
    const float c = cs.x, s = cs.y;
    const int D = g.depth;
    const float Xc = (float)X - g.cx;
    const float ax = fmaf(Xc, c, g.hx);
    const float ay = fmaf(Xc, -s, g.hy);
    // the samples whose base texel lies in [-1, n-1] in x and in y: one limit per lane of the ray
    const bool bound_x = ph < 2, upper = (ph & 1) != 0;
    int v = 0;
    if (X < g.px) {
        const float a = bound_x ? ax : ay, sl = bound_x ? s : c;
        const float hi = bound_x ? (float)g.nx : (float)g.ny;
        if (sl != 0.0f) v = first_true(((sl > 0.0f) != upper) ? -1.0f : hi, a, sl, 1.0f / sl, g.hd, D);
        else v = upper ? ((a >= -1.0f && a < hi) ? D : 0) : 0;
    }
    const int w = __shfl_xor_sync(0xffffffffu, v, 2);
    const int m = upper ? min(v, w) : max(v, w);
    const int u = __shfl_xor_sync(0xffffffffu, m, 1);
    const int ya = upper ? u : m, yb = upper ? m : u;
    xct_grid_wait();
    xct_grid_trigger();
    const float *im = img + (size_t)z * g.nx * g.ny;
    float sum = 0.0f;
#pragma unroll 4
    for (int Y = ya + warp * kDirLanes + ph; Y < yb; Y += W * kDirLanes) {
        const float Yc = (float)Y - g.hd;
        const float x = fmaf(Yc, s, ax), y = fmaf(Yc, c, ay);
        const float tx = __fadd_rd(x, kMagic), ty = __fadd_rd(y, kMagic);  // floor in the low bits
        const int i = __float_as_int(tx) - XCT_FLOOR_BIAS, j = __float_as_int(ty) - XCT_FLOOR_BIAS;
        const float fx = x - (tx - kMagic), fy = y - (ty - kMagic);
        const bool i0 = i >= 0, i1 = i + 1 < g.nx, j0 = j >= 0, j1 = j + 1 < g.ny;
        const float *r0 = im + (j * g.nx + i);
        const float t00 = (i0 && j0) ? r0[0] : 0.0f;
        const float t10 = (i1 && j0) ? r0[1] : 0.0f;
        const float t01 = (i0 && j1) ? r0[g.nx] : 0.0f;
        const float t11 = (i1 && j1) ? r0[g.nx + 1] : 0.0f;
        sum += xct_lerp(fy, xct_lerp(fx, t00, t10), xct_lerp(fx, t01, t11));
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if (ph == 0) part[warp][ray] = sum;
    __syncthreads();
    if (warp != 0) return;
    // the warps' partial sums in double: lane ph of a ray takes every fourth
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < W; q += kDirLanes)
        if (q + ph < W) t += (double)part[q + ph][ray];
    t += __shfl_xor_sync(0xffffffffu, t, 1);
    t += __shfl_xor_sync(0xffffffffu, t, 2);
    if (ph == 0 && X < g.px) {
        const float p = (float)t;
        const size_t o = ((size_t)z * g.pa + th) * g.px + X;
        out[o] = meas != nullptr ? xct_ratio(xct_measured(meas + (size_t)z * g.pa * g.px, g.px, g.pa, X, th, g.fetch), p) : p;
    }
}

// grid: (ceil(nx / 32), ceil(ny / 4), ceil(dN / S)), 128 threads.
template <int S>
__global__ void __launch_bounds__(128) bp_direct_kernel(float *img, const float *ratio,
                                                        const float2 *__restrict__ trig, KGeom g, int dN, int sub,
                                                        int nang, float ssf, float paf)
{
    const int X = (int)blockIdx.x * 32 + (int)(threadIdx.x & 31), Y = (int)blockIdx.y * 4 + (int)(threadIdx.x >> 5);
    const int z0 = (int)blockIdx.z * S;
    xct_grid_wait();
    xct_grid_trigger();
    if (X >= g.nx || Y >= g.ny) return;
    const size_t nprj = (size_t)g.pa * g.px;
    const float Xc = (float)X - g.hx, Yc = (float)Y - g.hy;
    const float *row = ratio + (size_t)z0 * nprj + (size_t)sub * g.px;
    const float2 *tr = trig + sub;
    const bool two = S == 2 && z0 + 1 < dN;
    float b[S];
#pragma unroll
    for (int q = 0; q < S; ++q) b[q] = 0.0f;
    const size_t zoff = two ? nprj : 0;
    const size_t rstep = (size_t)g.ss * g.px;
#pragma unroll 6
    for (int k = 0; k < nang; ++k, row += rstep, tr += g.ss) {
        const float2 cs = __ldg(tr);
        const int bin = xct_floor_bits(xct_bin_coord(Xc, cs.x, Yc * cs.y, g.cx)) - XCT_FLOOR_BIAS;
        const bool in = (unsigned)bin < (unsigned)g.px;
        b[0] += in ? row[bin] : 0.0f;
        if (S == 2) b[S - 1] += in ? row[zoff + bin] : 0.0f;
    }
    float *p = img + ((size_t)z0 * g.ny + Y) * g.nx + X;
    *p = xct_update(*p, b[0], ssf, paf);
    if (two) {
        p += (size_t)g.nx * g.ny;
        *p = xct_update(*p, b[S - 1], ssf, paf);
    }
}

}  // namespace

// a tile or a switch set by hand holds whatever the size
static bool by_hand(const KGeom &g) { return g.fwd_hand || g.ms_hand; }

bool fwd_is_direct(const KGeom &g, int dN, int nrows)
{
    return !by_hand(g) && (long long)g.nx * g.ny * nrows * dN <= kDirectTaps && nrows <= 65535 && dN <= kMaxGridZ;
}

bool bp_is_direct(const KGeom &g, int dN)
{
    return !by_hand(g) && (long long)g.nx * g.ny * dN <= kDirectPixels && dN <= kMaxGridZ;
}

int launch_fwd_direct(const KGeom &g, const float2 *trig, const float *img, const float *meas, float *out, int dN, int sub,
                      int step, int nrows, cudaStream_t st)
{
    if (nrows <= 0 || dN <= 0) return XCT_OK;
    const dim3 grid((g.px + kDirRays - 1) / kDirRays, nrows, dN);
    return xct_launch(fwd_direct_kernel, grid, kDirWarps * 32, 0, st, img, meas, out, trig, g, sub, step);
}

int launch_bp_update_direct(const KGeom &g, const float2 *trig, float *img, const float *ratio, int dN, int sub,
                            cudaStream_t st)
{
    if (dN <= 0) return XCT_OK;
    const int nang = (g.pa - sub + g.ss - 1) / g.ss;
    const dim3 grid((g.nx + 31) / 32, (g.ny + 3) / 4, dN >= 2 ? (dN + 1) / 2 : 1);
    if (dN >= 2)
        return xct_launch(bp_direct_kernel<2>, grid, 128, 0, st, img, ratio, trig, g, dN, sub, nang, (float)g.ss, (float)g.pa);
    return xct_launch(bp_direct_kernel<1>, grid, 128, 0, st, img, ratio, trig, g, dN, sub, nang, (float)g.ss, (float)g.pa);
}
