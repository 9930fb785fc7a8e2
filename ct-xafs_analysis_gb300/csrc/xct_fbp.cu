// xct_fbp.cu -- filtered backprojection and the base-up step of the FBP + OS-EM hybrid.
//
// Replaces, for CT_reconstruction:
//   FBP_execution (GPU.cpp:665-819) over the kernels of FBP.cl:
//     spinFactor .. outputImage (FBP.cl:34-160)  -> fbp_filter_kernel (one launch)
//     backProjectionFBP (FBP.cl:164-188)          -> fbp_bp_ms_kernel
//   hybrid_thread's base-up (GPU.cpp:1538-1566):
//     findMinimumX/findMinimumY (reconstShare.cl:111-177) -> folded into fbp_bp_ms_kernel
//     baseUp (reconstShare.cl:87-109)                     -> base_up_kernel
//
// Ramp filter.  The reference zero-pads each sinogram row to ZP_SIZE bins, runs a radix-2
// FFT in global memory (one launch per butterfly stage), multiplies by the ramp
// |k| * PI/ZP_SIZE, runs the inverse FFT the same way and keeps the real part.  Here one
// CTA filters two rows a, b at once in shared memory: z = a + i b, Z = FFT(z),
// Y = Z * H / zp, y = IFFT(Y) = filt(a) + i filt(b), which holds because the ramp H is real
// and even.  The transform is a Stockham autosort FFT (radix 8, then 4 or 2), the inverse is
// taken as conj(FFT(conj(Y))).  The reference moves bin px/2 to index 0 before the
// transform (FBP.cl:53-56); a circular shift commutes with a circular convolution, so the
// bins stay in place here and the filtered row is the same in exact arithmetic.  The
// rounding differs from the reference's radix-2 float FFT at the 1e-6 relative level.
//
// FBP backprojection.  The OS-EM backprojector's tiling (32 x 32 pixels of up to eight slices,
// per-angle windows of the filtered rows staged in shared memory), with the
// reference's linear sampler along the row and its per-pixel expression order, so the
// image is bit-identical to FBP.cl's for the same filtered sinogram.
#include <math.h>
#include <stdio.h>

#include <algorithm>
#include <type_traits>

#include "xct_async.cuh"
#include "xct_check.cuh"
#include "xct_device.cuh"
#include "xct_f32x2.cuh"
#include "xct_internal.h"

namespace {

// ------------------------------------------------------------------ ramp filter (FFT)
__device__ __forceinline__ int fpad(int i) { return i + (i >> 4); }  // 16-entry rows + 1

__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul_mi(float2 a) { return make_float2(a.y, -a.x); }  // a * (-i)

// Forward DFT of R points in registers: y[k] = sum_r v[r] exp(-2 pi i r k / R).
__device__ __forceinline__ void dft2(float2 &a, float2 &b)
{
    const float2 t = a;
    a = cadd(t, b);
    b = csub(t, b);
}
__device__ __forceinline__ void dft4(float2 &v0, float2 &v1, float2 &v2, float2 &v3)
{
    const float2 t0 = cadd(v0, v2), t1 = csub(v0, v2), t2 = cadd(v1, v3), t3 = cmul_mi(csub(v1, v3));
    v0 = cadd(t0, t2);
    v2 = csub(t0, t2);
    v1 = cadd(t1, t3);
    v3 = csub(t1, t3);
}
template <int R>
__device__ __forceinline__ void dft(float2 *v)
{
    if constexpr (R == 2) {
        dft2(v[0], v[1]);
    } else if constexpr (R == 4) {
        dft4(v[0], v[1], v[2], v[3]);
    } else {
        // 8 = 2 x 4: DFT4 of the even and the odd samples, then the W8^k combination
        float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
        float2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
        dft4(e0, e1, e2, e3);
        dft4(o0, o1, o2, o3);
        const float h = 0.70710678118654752f;
        o1 = make_float2((o1.x + o1.y) * h, (o1.y - o1.x) * h);   // * (1 - i)/sqrt2
        o2 = cmul_mi(o2);                                         // * (-i)
        o3 = make_float2((o3.y - o3.x) * h, -(o3.x + o3.y) * h);  // * (-1 - i)/sqrt2
        v[0] = cadd(e0, o0);
        v[4] = csub(e0, o0);
        v[1] = cadd(e1, o1);
        v[5] = csub(e1, o1);
        v[2] = cadd(e2, o2);
        v[6] = csub(e2, o2);
        v[3] = cadd(e3, o3);
        v[7] = csub(e3, o3);
    }
}

// One Stockham pass of radix R over xs[zp] (padded): butterfly j < zp/R reads
// xs[j + r*zp/R], twiddles by exp(-2 pi i r k / (Ns R)) with k = j mod Ns, transforms, and
// writes xs[(j - k) R + k + r Ns].  Each thread owns VPT/R butterflies; all reads finish
// before the barrier, so the pass is in place.
template <int R, int VPT>
__device__ __forceinline__ void stockham_pass(float2 *xs, int zp, int Ns, float tscale)
{
    constexpr int B = VPT / R;
    const int T = blockDim.x, stride = zp / R;
    float2 v[B][R];
#pragma unroll
    for (int q = 0; q < B; ++q) {
        const int j = threadIdx.x + q * T;
        const int k = j & (Ns - 1);
#pragma unroll
        for (int r = 0; r < R; ++r) v[q][r] = xs[fpad(j + r * stride)];
        if (Ns > 1) {
            // angle 2 pi r k / (Ns R) = pi * (2 r k zp/(Ns R)) / zp; tscale = 2 / (Ns R)
#pragma unroll
            for (int r = 1; r < R; ++r) {
                float s, c;
                sincospif((float)(r * k) * tscale, &s, &c);
                v[q][r] = cmul(v[q][r], make_float2(c, -s));
            }
        }
        dft<R>(v[q]);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < B; ++q) {
        const int j = threadIdx.x + q * T;
        const int k = j & (Ns - 1);
        const int d = (j - k) * R + k;
#pragma unroll
        for (int r = 0; r < R; ++r) xs[fpad(d + r * Ns)] = v[q][r];
    }
    __syncthreads();
}

template <int VPT>
__device__ __forceinline__ void fft_forward(float2 *xs, int zp, int logzp)
{
    int Ns = 1, rem = logzp;
    while (rem > 0) {
        if (VPT >= 8 && rem >= 3) {
            stockham_pass<(VPT >= 8 ? 8 : 2), VPT>(xs, zp, Ns, 2.0f / (float)(Ns * 8));
            Ns <<= 3;
            rem -= 3;
        } else if (VPT >= 4 && rem >= 2) {
            stockham_pass<(VPT >= 4 ? 4 : 2), VPT>(xs, zp, Ns, 2.0f / (float)(Ns * 4));
            Ns <<= 2;
            rem -= 2;
        } else {
            stockham_pass<2, VPT>(xs, zp, Ns, 2.0f / (float)(Ns * 2));
            Ns <<= 1;
            rem -= 1;
        }
    }
}

// grid: ceil(nrows / 2) CTAs of zp / VPT threads (at least 32); rows 2c and 2c+1 of the
// flattened [nrows][px] sinogram stack.  h = PI/zp as the reference stores it (a float).
template <int VPT>
__global__ void __launch_bounds__(1024) fbp_filter_kernel(const float *__restrict__ sino, float *__restrict__ out,
                                                          long long nrows, int px, int zp, int logzp, float h)
{
    extern __shared__ float2 xs[];
    const int T = blockDim.x;
    const long long r0 = 2LL * blockIdx.x;
    const bool has_b = r0 + 1 < nrows;
    const float *ra = sino + r0 * px;
    for (int n = threadIdx.x; n < zp; n += T) {
        float a = 0.0f, b = 0.0f;
        if (n < px) {
            a = __ldg(ra + n);
            if (has_b) b = __ldg(ra + px + n);
        }
        xs[fpad(n)] = make_float2(a, b);
    }
    __syncthreads();
    fft_forward<VPT>(xs, zp, logzp);
    // ramp (FBP.cl:132-133: X*h below zp/2, (zp - X)*h above), then conj for the inverse
    for (int k = threadIdx.x; k < zp; k += T) {
        const float f = (float)min(k, zp - k) * h;
        const float2 v = xs[fpad(k)];
        xs[fpad(k)] = make_float2(v.x * f, -(v.y * f));
    }
    __syncthreads();
    fft_forward<VPT>(xs, zp, logzp);
    // y = conj(F) / zp (a power of two: the scaling is exact)
    const float inv = 1.0f / (float)zp;
    float *oa = out + r0 * px;
    for (int n = threadIdx.x; n < px; n += T) {
        const float2 v = xs[fpad(n)];
        oa[n] = v.x * inv;
        if (has_b) oa[px + n] = -v.y * inv;
    }
}

// ------------------------------------------------------------ FBP backprojection
// Monotone integer key of a float (atomicMin on keys orders as the floats do).
__device__ __forceinline__ int fkey(float f)
{
    const int b = __float_as_int(f);
    return b >= 0 ? b : b ^ 0x7FFFFFFF;
}
__device__ __forceinline__ float fkey_decode(int k) { return __int_as_float(k >= 0 ? k : k ^ 0x7FFFFFFF); }

// img[Y][X] = (1/(2 pa)) sum_th lin(fprj[th], u) for pixels with r < nx/2, else 0
// (FBP.cl:178-187); u = ((Xc c - Yc s) + cx) + 0.5, sampled by the linear
// sampler at (u, th + 0.5): i = floor(u - 0.5), a = (u - 0.5) - i,
// (1 - a) t[i] + a t[i+1], zero off the detector.  min_keys (optional): the per-slice
// minimum of the written image, as keys.
//
// For the slices of one call (one geometry) a (pixel, angle) pair reads the same two bins in
// all slices of a group, so the bin coordinate, floor and fraction are found once for
// S lerps.  A CTA of 256 threads owns a 32 x 32 pixel tile of S slices (8, 2 or 1) and stages the
// window of the tile's bins (< 49 with the lerp's second bin, bounded exactly by the tile corners -- the
// coordinate is monotone in X and in Y -- its start rounded down to a multiple of 4) by asynchronous
// copies, a chunk of angles at a time: per slice pair as (t_z, t_z+1) pairs, for one slice as
// (t[j], t[j+1]) pairs, so that its lerp is one 64-bit load.  A thread takes 4 pixels of one row (8 apart);
// per pixel and angle the literal expression for u (products and differences in scalar: ptxas fuses a
// packed multiply feeding a packed add or subtract, and the reference rounds each operation), floor as
// a round-down add, the products in scalar, sums and accumulation packed over the slice pair (over the
// pixel pair for one slice), in angle order, so every form gives a slice the same bits.
//
// A warp whose 32 x 4 pixels all lie outside the field of view (their values are 0 whatever the
// projections) skips its gathers: 20 % of a square image.
//
// Bound: the FP32 pipe for one slice (13 operations a lerp that the reference's rounding fixes), the
// shared-memory data path for eight (8 B per lerp and slice).  One 2048^2 slice, 1500 angles: 2.49 ms (2.51 with
// that pipe 72 % busy, rows of tiles from the top down; 2.88 with 64 x 64 tiles that covered the whole square).
constexpr int kFbpMsT = 32, kFbpMsThreads = 256, kFbpMsW = 52, kFbpMsPix = 4, kFbpMsSlices = 8;

template <int S>
struct FbpMsShared {
    static constexpr int P = S == 1 ? 1 : S / 2;           // pairs per bin
    static constexpr int Chunk = S == 8 ? 24 : 48;         // angles per staging pass
    static constexpr unsigned PairBytes = (unsigned)(Chunk * kFbpMsW * 8);  // one pair's windows
    float2 win[P * Chunk * kFbpMsW];  // [pair][angle][bin]
    float2 scs[Chunk];
    int slo[Chunk];
    unsigned soff[Chunk];  // shared address of angle k's entry for floor bits fb: soff[k] + 8*fb
    float red[kFbpMsThreads / 32][S];
};

// Both bins of slice pair H .. P-1 at byte address ad, weighted and added to the pairs' sums.
template <int S, int H = 0>
__device__ __forceinline__ void fbp_pairs(unsigned ad, float w, float a, f2x *acc)
{
    if constexpr (H < S / 2) {
        float t0a, t0b, t1a, t1b;  // (slice 2H, 2H+1) at bins i and i + 1
        lds_f2_at<(int)(H * FbpMsShared<S>::PairBytes)>(ad, t0a, t0b);
        lds_f2_at<(int)(H * FbpMsShared<S>::PairBytes + 8)>(ad, t1a, t1b);
        const float pa0 = w * t0a, pb0 = w * t0b, pa1 = a * t1a, pb1 = a * t1b;
        acc[H] = f2_add(acc[H], f2_add(f2_pack(pa0, pb0), f2_pack(pa1, pb1)));
        fbp_pairs<S, H + 1>(ad, w, a, acc);
    }
}

// grid: (ntx * nty tiles of 32 x 32, 1, dN / S slice groups).
template <int S>
__global__ void __launch_bounds__(kFbpMsThreads) fbp_bp_ms_kernel(const float *__restrict__ fprj,
                                                                  float *__restrict__ img,
                                                                  const float2 *__restrict__ trig, KGeom g, int ntx,
                                                                  int *__restrict__ min_keys)
{
    typedef FbpMsShared<S> C;
    constexpr int kAcc = S == 1 ? kFbpMsPix / 2 : kFbpMsPix * C::P;
    __shared__ __align__(16) C sh;
    const int z0 = (int)blockIdx.z * S;
    const size_t nprj = (size_t)g.pa * g.px, nimg = (size_t)g.nx * g.ny;
    const float *rz = fprj + (size_t)z0 * nprj;
    // rows of tiles from the middle outwards: the last CTAs to start are the rows whose corners have nothing to do
    const int row = (int)blockIdx.x / ntx, mid = ((int)gridDim.x / ntx - 1) / 2;
    const int bx = (int)blockIdx.x - row * ntx, by = row & 1 ? mid + (row + 1) / 2 : mid - row / 2;
    const int X0 = bx * kFbpMsT, Y0 = by * kFbpMsT;
    const int X1 = min(X0 + kFbpMsT, g.nx) - 1, Y1 = min(Y0 + kFbpMsT, g.ny) - 1;
    const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
    const float Yc = (float)min(Y0 + ty, Y1) - g.hy;
    float xc[kFbpMsPix];
#pragma unroll
    for (int i = 0; i < kFbpMsPix; ++i) xc[i] = (float)min(X0 + tx + 8 * i, X1) - g.hx;
    f2x acc[kAcc];  // S > 1: [pixel][slice pair]; S = 1: pixel pairs
#pragma unroll
    for (int i = 0; i < kAcc; ++i) acc[i] = 0ull;
    // any pixel of this warp inside the field of view (the epilogue's own test)
    bool in_view = false;
#pragma unroll
    for (int i = 0; i < kFbpMsPix; ++i) in_view |= sqrtf(xc[i] * xc[i] + Yc * Yc) < g.hx;
    in_view = __any_sync(0xffffffffu, in_view);
    const unsigned wbase = (unsigned)__cvta_generic_to_shared(sh.win);
    const f2x cxp = f2_pack(g.cx, g.cx), hp = f2_pack(0.5f, 0.5f), MM = f2_pack(12582912.0f, 12582912.0f);
    const f2x one2 = f2_pack(1.0f, 1.0f);
    const int nang = __syncthreads_or(in_view) ? g.pa : 0;  // a tile outside the field of view stages nothing
    for (int k0 = 0; k0 < nang; k0 += C::Chunk) {
        const int kn = min(C::Chunk, g.pa - k0);
        __syncthreads();
        for (int k = threadIdx.x; k < kn; k += kFbpMsThreads) {
            const float2 cs = trig[k0 + k];
            sh.scs[k] = cs;
            const float xa = (float)X0 - g.hx, xb = (float)X1 - g.hx;
            const float qa = ((float)Y0 - g.hy) * cs.y, qb = ((float)Y1 - g.hy) * cs.y;
            int lo = xct_floor_bits(xct_bin_coord(xa, cs.x, qa, g.cx) - 0.5f);
            lo = min(lo, xct_floor_bits(xct_bin_coord(xb, cs.x, qa, g.cx) - 0.5f));
            lo = min(lo, xct_floor_bits(xct_bin_coord(xa, cs.x, qb, g.cx) - 0.5f));
            lo = min(lo, xct_floor_bits(xct_bin_coord(xb, cs.x, qb, g.cx) - 0.5f));
            lo &= ~3;  // the bias is a multiple of 4: this rounds the bin down to one
            sh.slo[k] = lo - XCT_FLOOR_BIAS;
            sh.soff[k] = wbase + 8u * (unsigned)(k * kFbpMsW) - 8u * (unsigned)lo;
        }
        __syncthreads();
        // S > 1: window (pair p, angle k, bin lo_k + r) = (t_{2p}, t_{2p+1}); S = 1: (t[r], t[r + 1]); 0 off
        // the detector
        if constexpr (S == 1) {
            for (int e = threadIdx.x; e < kn * kFbpMsW; e += kFbpMsThreads) {
                const int r = e % kFbpMsW, k = e / kFbpMsW;
                const int bin = sh.slo[k] + r;
                const float *row = rz + (size_t)(k0 + k) * g.px;
                const bool i0 = (unsigned)bin < (unsigned)g.px, i1 = (unsigned)(bin + 1) < (unsigned)g.px;
                const unsigned dst = wbase + 8u * (unsigned)e;
                cp_async4(dst, i0 ? (const void *)(row + bin) : (const void *)row, i0 ? 4u : 0u);
                cp_async4(dst + 4u, i1 ? (const void *)(row + bin + 1) : (const void *)row, i1 ? 4u : 0u);
            }
        } else {
            for (int e = threadIdx.x; e < kn * S * kFbpMsW; e += kFbpMsThreads) {
                const int r = e % kFbpMsW, t2 = e / kFbpMsW;
                const int z = t2 % S, k = t2 / S;
                const int bin = sh.slo[k] + r;
                const float *row = rz + (size_t)z * nprj + (size_t)(k0 + k) * g.px;
                const bool in = (unsigned)bin < (unsigned)g.px;
                const unsigned dst =
                    wbase + (unsigned)(z >> 1) * C::PairBytes + 8u * (unsigned)(k * kFbpMsW + r) + 4u * (unsigned)(z & 1);
                cp_async4(dst, in ? (const void *)(row + bin) : (const void *)row, in ? 4u : 0u);
            }
        }
        cp_async_wait_all();
        __syncthreads();
        // any entry whose next entry (the lerp's second bin) is staged
        const unsigned wlo = wbase, whi = wbase + 8u * (unsigned)(kn * kFbpMsW - (S == 1 ? 1 : 2));
        (void)wlo;
        (void)whi;
        if (!in_view) continue;
        for (int k = 0; k < kn; ++k) {
            const float c = sh.scs[k].x, s = sh.scs[k].y;
            const unsigned off = sh.soff[k];
            const float q = Yc * s;
#pragma unroll
            for (int j = 0; j < kFbpMsPix / 2; ++j) {
                // uu = (((Xc*c - q) + cx) + 0.5) - 0.5, fi = floor(uu), a = uu - fi for pixels 2j and 2j+1
                const float p0 = xc[2 * j] * c, p1 = xc[2 * j + 1] * c;
                const f2x d = f2_pack(p0 - q, p1 - q);
                const f2x uu = f2_sub(f2_add(f2_add(d, cxp), hp), hp);
                const f2x tb = f2_add_rd(uu, MM);
                const f2x a2 = f2_sub(uu, f2_sub(tb, MM));
                const f2x w2 = f2_sub(one2, a2);
                int e0, e1;
                f2_unpack_bits(tb, e0, e1);
                float a[2], w[2];
                f2_unpack(a2, a[0], a[1]);
                f2_unpack(w2, w[0], w[1]);
                const unsigned ad[2] = {(unsigned)e0 * 8u + off, (unsigned)e1 * 8u + off};
                if constexpr (S == 1) {
                    float t[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                        if (XCT_IN(ad[u], wlo, whi, XCT_SITE_FBP_WIN)) lds_f2_at<0>(ad[u], t[u][0], t[u][1]);
                    const float p00 = w[0] * t[0][0], p01 = a[0] * t[0][1];
                    const float p10 = w[1] * t[1][0], p11 = a[1] * t[1][1];
                    acc[j] = f2_add(acc[j], f2_add(f2_pack(p00, p10), f2_pack(p01, p11)));
                } else {
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        if (!XCT_IN(ad[u], wlo, whi, XCT_SITE_FBP_WIN)) continue;
                        fbp_pairs<S>(ad[u], w[u], a[u], acc + (2 * j + u) * C::P);
                    }
                }
            }
        }
    }
    const float two_pa = (float)g.pa * 2.0f;
    const int Y = Y0 + ty;
    float vmin[S];
#pragma unroll
    for (int z = 0; z < S; ++z) vmin[z] = INFINITY;
    if (Y <= Y1) {
#pragma unroll
        for (int i = 0; i < kFbpMsPix; ++i) {
            const int X = X0 + tx + 8 * i;
            if (X > X1) continue;
            const float rr = sqrtf(xc[i] * xc[i] + Yc * Yc);
#pragma unroll
            for (int z = 0; z < S; ++z) {
                float v2[2];
                f2_unpack(S == 1 ? acc[i / 2] : acc[i * C::P + z / 2], v2[0], v2[1]);
                const float v = (rr < g.hx) ? __fdiv_rn(v2[S == 1 ? i & 1 : z & 1], two_pa) : 0.0f;
                img[(size_t)(z0 + z) * nimg + (size_t)Y * g.nx + X] = v;
                vmin[z] = fminf(vmin[z], v);
            }
        }
    }
    if (min_keys != nullptr) {
#pragma unroll
        for (int z = 0; z < S; ++z) {
            float m = vmin[z];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = fminf(m, __shfl_xor_sync(0xffffffffu, m, o));
            if ((threadIdx.x & 31) == 0) sh.red[threadIdx.x >> 5][z] = m;
        }
        __syncthreads();
        if (threadIdx.x < S) {
            float m = sh.red[0][threadIdx.x];
            for (int i = 1; i < kFbpMsThreads / 32; ++i) m = fminf(m, sh.red[i][threadIdx.x]);
            atomicMin(min_keys + z0 + threadIdx.x, fkey(m));
        }
    }
}

// baseUp (reconstShare.cl:87-109) over dN slices of n pixels, in place, a = the slice
// minimum: b1 = (v - a)/a (0 when a == 0); g = sum_{i<=order} (-1)^(i+1) b1^i / i in float;
// v -= a * exp(g).
__global__ void base_up_kernel(float *__restrict__ img, long long n, int dN, int order,
                               const int *__restrict__ min_keys)
{
    const long long total = n * dN;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const float a = fkey_decode(__ldg(min_keys + idx / n));
        const float v = img[idx];
        float gs = 0.0f;
        const float b1 = (a != 0.0f) ? __fdiv_rn(v - a, a) : 0.0f;
        float b2 = 1.0f, flag = -1.0f;
        for (int i = 1; i <= order; ++i) {
            b2 *= b1;
            flag *= -1.0f;
            gs += __fdiv_rn(flag * b2, (float)i);
        }
        img[idx] = v - a * expf(gs);
    }
}

int fbp_vpt(int zp) { return zp >= 16384 ? 16 : (zp >= 256 ? 8 : zp / 32); }

template <int VPT>
int launch_filter_vpt(const float *sino, float *out, long long nrows, int px, int zp, int logzp, float h,
                      cudaStream_t st)
{
    const int threads = zp / VPT;
    const size_t smem = sizeof(float2) * (size_t)(zp + zp / 16);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(fbp_filter_kernel<VPT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return xct_cuda_fail(e, "fbp_filter smem attribute");
    }
    const long long ctas = (nrows + 1) / 2;
    if (ctas > 0x7FFFFFFFLL) return xct_fail(XCT_E_INVALID, "fbp filter: too many rows in one call");
    fbp_filter_kernel<VPT><<<(unsigned)ctas, threads, smem, st>>>(sino, out, nrows, px, zp, logzp, h);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return xct_cuda_fail(e, "fbp_filter_kernel launch");
    g_xct_launches.fetch_add(1);
    return XCT_OK;
}

}  // namespace

int xct_fbp_check_zp(int px, int &zp)
{
    if (zp == 0) {
        zp = 1;
        while (zp < 2 * px) zp *= 2;
    }
    if (zp < 64 || zp > 16384 || (zp & (zp - 1)) != 0 || zp < px) {
        char b[200];
        snprintf(b, sizeof b,
                 "fbp: zero padding %d must be a power of two in [64, 16384] and >= the detector width %d", zp, px);
        return xct_fail(XCT_E_INVALID, b);
    }
    return XCT_OK;
}

int launch_fbp_filter(const KGeom &g, const float *sino, float *out, int dN, int zp, cudaStream_t st)
{
    int logzp = 0;
    while ((1 << logzp) < zp) ++logzp;
    const float h = (float)(3.14159265358979323846 / zp);  // FBP.cl:132
    const long long nrows = (long long)dN * g.pa;
    switch (fbp_vpt(zp)) {
    case 2: return launch_filter_vpt<2>(sino, out, nrows, g.px, zp, logzp, h, st);
    case 4: return launch_filter_vpt<4>(sino, out, nrows, g.px, zp, logzp, h, st);
    case 8: return launch_filter_vpt<8>(sino, out, nrows, g.px, zp, logzp, h, st);
    default: return launch_filter_vpt<16>(sino, out, nrows, g.px, zp, logzp, h, st);
    }
}

int launch_fbp_bp(const KGeom &g, const float2 *trig, const float *fprj, float *img, int dN, int *min_keys,
                  cudaStream_t st)
{
    if (min_keys != nullptr) {
        cudaError_t e = cudaMemsetAsync(min_keys, 0x7F, sizeof(int) * dN, st);  // key of a huge float
        if (e != cudaSuccess) return xct_cuda_fail(e, "fbp min reset");
    }
    // Slices go in groups of eight (with the slice-interleaved kernels on), pairs (with grouping on) and singles, as
    // the modelled time of the launches, one after the other, is least: us an angle of a launch whose SMs get m CTAs
    // each, a + c m (fits of 64^2 to 2048^2).  The larger forms take less per slice and more per CTA, and each further
    // launch another a: three slices of 400^2 x 200 angles 69 us as singles and 89 as a pair and one, of 1024^2 x 512
    // 668 and 578.  Eights set by hand hold whatever the size.
    const int mtx = (g.nx + kFbpMsT - 1) / kFbpMsT, mty = (g.ny + kFbpMsT - 1) / kFbpMsT;
    const long long tiles = (long long)mtx * mty;
    const int sms = device_sm_count();
    auto time = [&](double a, double c, int groups) { return groups > 0 ? a + c * (double)((tiles * groups + sms - 1) / sms) : 0.0; };
    int eights = 0, pairs = 0;
    double least = INFINITY;
    for (int e = 0; e <= (g.ms_chunk > 0 ? dN / kFbpMsSlices : 0); e += std::max(1, dN / kFbpMsSlices)) {
        if (e == 0 && g.ms_hand && g.ms_chunk > 0 && dN >= kFbpMsSlices) continue;
        for (int two = 0; two <= (g.fwd_group ? 1 : 0); ++two) {
            const int rest = dN - e * kFbpMsSlices, p = two ? rest / 2 : 0;
            const double t = time(0.2, 0.25, e) + time(0.095, 0.085, p) + time(0.07, 0.062, rest - 2 * p);
            if (t < least) least = t, eights = e, pairs = p;
        }
    }
    auto run = [&](auto sc, int groups) -> int {
        constexpr int S = decltype(sc)::value;
        if (groups <= 0) return XCT_OK;
        fbp_bp_ms_kernel<S><<<dim3(mtx * mty, 1, groups), kFbpMsThreads, 0, st>>>(fprj, img, trig, g, mtx, min_keys);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return xct_cuda_fail(e, "fbp_bp_ms_kernel launch");
        g_xct_launches.fetch_add(1);
        fprj += (size_t)groups * S * g.pa * g.px;
        img += (size_t)groups * S * g.nx * g.ny;
        if (min_keys != nullptr) min_keys += groups * S;
        dN -= groups * S;
        return XCT_OK;
    };
    int rc = run(std::integral_constant<int, kFbpMsSlices>{}, eights);
    if (!rc) rc = run(std::integral_constant<int, 2>{}, pairs);
    if (!rc) rc = run(std::integral_constant<int, 1>{}, dN);
    return rc;
}

int launch_base_up(const KGeom &g, float *img, int dN, int order, const int *min_keys, int sm_count, cudaStream_t st)
{
    const long long n = (long long)g.nx * g.ny;
    const long long want = (n * dN + 255) / 256;
    const int blocks = (int)std::min<long long>(want, (long long)sm_count * 8);
    base_up_kernel<<<blocks, 256, 0, st>>>(img, n, dN, order, min_keys);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return xct_cuda_fail(e, "base_up_kernel launch");
    g_xct_launches.fetch_add(1);
    return XCT_OK;
}

XCT_CHECK_READER(xct_check_read_fbp)
