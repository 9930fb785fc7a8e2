// xct_tiled.cu -- the optimised OS-EM kernels for sm_103a.
//
// Forward projector (OSEM1 / projection, OSEM.cl:38-68, reconstShare.cl:213-241),
// tile-stationary:
//   * one CTA owns an image tile of up to five slices: the samples whose base texel (floor(x),
//     floor(y)) lies in [x0, x0+tx) x [y0, y0+ty), tx, ty <= T, the first at -1 (base texel -1 still
//     reaches texel 0).  It stages the tile once in shared memory as (t, t[x+1] - t) pairs, so
//     the x-lerp of a bilinear sample is one FMA and its 2x2 footprint is two 64-bit
//     loads, and serves its angles from there; a run of (tile, angle) units of equal modelled time per
//     CTA, so that the grid is one wave (slices of up to 4096 tiles; more, tiles set by hand and the batch
//     plans take a CTA per tile and chunk of angles);
//   * a warp takes one angle and 8 consecutive rays, 4 lanes per ray; the exact interval of
//     sample indices Y whose base texel lies in the tile (the coordinates are monotone in Y)
//     comes from four boundary searches, one per lane of the ray's group; the 4 lanes then
//     take every 4th sample, all rays in step from the warp's first sample on, with packed f32x2
//     coordinate/floor/fraction arithmetic over two samples;
//   * per-tile partial ray sums go into a double-precision accumulator with one atomic per
//     ray, slice and tile.
// A finalize kernel turns the accumulator into the OSEM1 ratio (or the raw projection)
// and clears it for the next subset.
//
// Backprojector (OSEM2, OSEM.cl:71-105), footprint-staged:
//   * one CTA owns a pixel tile (32x32 of up to eight slices); per
//     angle it stages the window of ratio bins its pixels hit (bin coordinates are monotone in X and in
//     Y, so the tile corners bound the window exactly) into shared memory;
//   * each thread gathers its pixels' bins per angle, in angle order, evaluating the
//     reference's bin expression ((Xc*c - Yc*s) + cx) + 0.5 with packed f32x2 instructions (each
//     lane rounds exactly like the scalar expression) and the nearest rule as a round-down add;
//   * the multiplicative update is fused.
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "xct_async.cuh"
#include "xct_check.cuh"
#include "xct_device.cuh"
#include "xct_f32x2.cuh"
#include "xct_launch.cuh"
#include "xct_ray.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kAngChunk = 128;  // most subset angles one forward-projector CTA serves

// A warp works on 8 consecutive rays of one angle with 4 lanes per ray, the 4 lanes taking
// every 4th sample (lane k: samples ya+k, ya+k+4, ...); 8 neighbouring rays have similar
// lengths inside a tile, so few lanes idle.
constexpr int kLanesPerRay = 4;
constexpr int kRaysPerWarp = 32 / kLanesPerRay;

constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23

__device__ __forceinline__ void lds_f2(unsigned addr, float &a, float &b)
{
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "r"(addr));
}
__device__ __forceinline__ float lds_f1(unsigned addr)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}

// ----------------------------------------------------------------- forward projector
// A CTA owns the samples whose base texel lies in a T x T tile of S slices (the slices of one call
// share their geometry, so a sample's coordinates, addresses and weights serve all S).  Shared
// memory holds one plane per slice of the elements (t(x), t(x+1) - t(x)), so a sample takes, per
// slice, two 64-bit loads (its two rows), two x-lerps and two weighted sums.
//
// Bound: the shared-memory data path, 16 B per sample and slice.  A 64-bit load is served a
// half-warp (4 rays x 4 samples here) at a time; with the rows loaded in image order the rotated
// lattice of a half-warp's samples collides in the banks whatever the pitch (a CPU model: 0.212
// wavefronts per sample at best, 0.125 ideal).  Loading the EVEN row of every sample's two first
// and the odd row second -- lanes whose base row is odd start with the row below -- halves the
// rows one load touches, and neighbouring samples then mostly share their elements: 0.127 with a
// pitch of 3 or 5 (mod 8).  The weight of the odd row is the distance |y - (even row)|.
//
// T: the side that fills shared memory with one CTA of 1024 threads per SM (163 for one slice, 83 for
// four), or with two of 512 (one stages while the other computes).  A larger tile has longer rays, so less
// of the time goes to finding a ray's interval and to its last, partly used step: per sample and slice
// 0.21 SM cycles against 0.26 for one slice (T = 163, 92), 0.147 against 0.167 for two (115, 83), 0.141
// against 0.148 for four (83, 58).  The sides 44, 60, 76 and 92 of one slice are a plan's choice by hand or by
// the tuner, and the batch plans'.
template <int S, int T>
struct FwdTile {
    // element pitch: the smallest of 3 or 5 (mod 8) that holds a row
    static constexpr int P = T % 8 <= 3 ? T - T % 8 + 3 : T % 8 <= 5 ? T - T % 8 + 5 : T - T % 8 + 11;
    static constexpr int Rows = T + 1;  // a base row r reads element rows r and r+1
    static constexpr unsigned Plane = (unsigned)(P * Rows * 8);
    // per chunk angle: (c, s, 1/c, 1/s) and (first ray, last ray, first item, end item)
    static constexpr size_t TableOff = ((size_t)S * Plane + 15) & ~(size_t)15;
    static constexpr size_t Smem = TableOff + (size_t)kAngChunk * 32;
    // large tiles: one CTA of 32 warps per SM; of S = 1, 12 warps per CTA, 4 CTAs per SM where four tiles
    // fit (T <= 76), else 3
    static constexpr bool Large = (Smem + 1024) * 2 > 228u * 1024u;
    static constexpr int Threads = Large ? 1024 : S == 1 && T <= 92 ? 384 : 512;
    static constexpr int MinBlocks = Large ? 1 : S > 1 || T > 92 ? 2 : (Smem + 1024) * 4 <= 228u * 1024u ? 4 : 3;
    static_assert((P % 8 == 3 || P % 8 == 5) && P >= T, "tile pitch");
    static_assert((Smem + 1024) * MinBlocks <= 228u * 1024u, "tiles exceed shared memory");
};
// Tile sides of the forms with S slices: the largest that one CTA per SM holds, and that two hold.
template <int S>
struct FwdGroup {
    static constexpr int Large = S == 1 ? 163 : S == 2 ? 115 : S == 3 ? 93 : S == 4 ? 83 : 75;
    static constexpr int T = S == 1 ? 115 : S == 2 ? 83 : S == 3 ? 67 : S == 4 ? 58 : 51;
};

template <int kOff>
__device__ __forceinline__ void lds_f2_off(unsigned addr, float &a, float &b)
{
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2+%3];" : "=f"(a), "=f"(b) : "r"(addr), "n"(kOff));
}

// Slices Z .. S-1 of one sample: its odd row's elements at B + kRow, its even row's at A + 2 kRow.
template <int S, unsigned kRow, unsigned Plane, int Z = 0>
__device__ __forceinline__ void fwd_tap(unsigned A, unsigned B, float fx, float wa, float wb, float (&sum)[S])
{
    if constexpr (Z < S) {
        float ta, da, tb, db;
        lds_f2_off<(int)(Z * Plane + 2 * kRow)>(A, ta, da);
        lds_f2_off<(int)(Z * Plane + kRow)>(B, tb, db);
        sum[Z] = fmaf(wa, fmaf(fx, da, ta), sum[Z]);
        sum[Z] = fmaf(wb, fmaf(fx, db, tb), sum[Z]);
        fwd_tap<S, kRow, Plane, Z + 1>(A, B, fx, wa, wb, sum);
    }
}

// Two samples of one ray at once, Yc = the halves of yc2 (f32x2 arithmetic, lane for lane the scalar
// one): coordinates x = fma(Yc, s, ax), y = fma(Yc, c, ay); floor(x) as a round-down add of 1.5*2^23;
// 2 floor(y/2) -- the even row at or above y -- as a round-down add of 1.5*2^24 (spacing 2).  With e =
// y - (that row + 1) in [-1, 1): the odd row is that row + 1, weight 1 - |e|; the even one is that row
// (e < 0) or the row below the odd one (e >= 0), weight |e|.  Pred: only where on0 / on1 are set.
// [alo, ahi]: the byte addresses a load may take (checked in the bounds-checked build only).
template <int S, int T, bool Pred>
__device__ __forceinline__ void fwd_pair(f2x yc2, f2x s2, f2x c2, f2x ax2, f2x ay2, f2x M23, f2x M24, f2x one2,
                                         unsigned base2, bool on0, bool on1, unsigned alo, unsigned ahi, float (&sum)[S])
{
    constexpr unsigned kRow = FwdTile<S, T>::P * 8, Plane = FwdTile<S, T>::Plane;
    const f2x x2 = f2_fma(yc2, s2, ax2), y2 = f2_fma(yc2, c2, ay2);
    const f2x tx = f2_add_rd(x2, M23), ty = f2_add_rd(y2, M24);
    const f2x fx2 = f2_sub(x2, f2_sub(tx, M23));
    const f2x e2 = f2_sub(y2, f2_add(f2_sub(ty, M24), one2));  // from the odd row: exact where the weight is small
    int ix[2], jy[2];
    float fx[2], e[2];
    f2_unpack_bits(tx, ix[0], ix[1]);
    f2_unpack_bits(ty, jy[0], jy[1]);
    f2_unpack(fx2, fx[0], fx[1]);
    f2_unpack(e2, e[0], e[1]);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        if (Pred && !(q ? on1 : on0)) continue;
        const unsigned B = (unsigned)jy[q] * (2u * kRow) + ((unsigned)ix[q] * 8u + base2);
        const unsigned A = B + (unsigned)(__float_as_int(e[q]) >> 31) * (2u * kRow);
        if (!XCT_IN(A + 2 * kRow, alo, ahi, XCT_SITE_FWD_TAP) || !XCT_IN(B + kRow, alo, ahi, XCT_SITE_FWD_TAP)) continue;
        const float wa = fabsf(e[q]);
        fwd_tap<S, kRow, Plane>(A, B, fx[q], wa, 1.0f - wa, sum);
    }
}

// The sums of a ray's four lanes: lane ph of the four ends with slice ph's (S = 1: lane 0's; S = 5:
// lane 0 also has slice 4's in `fifth`).
template <int S>
__device__ __forceinline__ float fwd_reduce(const float (&sum)[S], int ph, float &fifth)
{
    float v;
    if constexpr (S == 1) {
        v = sum[0] + __shfl_xor_sync(0xffffffffu, sum[0], 1);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
    } else if constexpr (S == 2) {
        const bool odd = ph & 1;
        v = (odd ? sum[1] : sum[0]) + __shfl_xor_sync(0xffffffffu, odd ? sum[0] : sum[1], 1);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
    } else {
        const bool hi = ph & 2, odd = ph & 1;
        const float s3 = S > 3 ? sum[S > 3 ? 3 : 0] : 0.0f;
        const float k0 = (hi ? sum[2] : sum[0]) + __shfl_xor_sync(0xffffffffu, hi ? sum[0] : sum[2], 2);
        const float k1 = (hi ? s3 : sum[1]) + __shfl_xor_sync(0xffffffffu, hi ? sum[1] : s3, 2);
        v = (odd ? k1 : k0) + __shfl_xor_sync(0xffffffffu, odd ? k0 : k1, 1);
        if constexpr (S == 5) {
            fifth = sum[4] + __shfl_xor_sync(0xffffffffu, sum[4], 1);
            fifth += __shfl_xor_sync(0xffffffffu, fifth, 2);
        }
    }
    return v;
}

// The tile of S slices (slice z: image image(z), accumulator accum(z) [nrows][px]) whose base texels are
// [x0, x0+tx) x [y0, y0+ty) (tx, ty <= T), for the subset angles k0 .. k0+chunk-1 (chunk <= kAngChunk).
// Starts and ends with all threads in step.
template <int S, int T, class Image, class Accum>
__device__ __forceinline__ void fwd_tile(const KGeom &g, Image image, Accum accum, const float2 *__restrict__ trig,
                                         int sub, int step, int nrows, int x0, int y0, int tx, int ty, int k0,
                                         int chunk, unsigned char *smem_raw)
{
    typedef FwdTile<S, T> C;
    constexpr int kThr = C::Threads;
    float4 *s_cs = reinterpret_cast<float4 *>(smem_raw + C::TableOff);
    int4 *s_ray = reinterpret_cast<int4 *>(s_cs + kAngChunk);
    const int kn = min(chunk, nrows - k0);
    if (kn <= 0) return;

    // element (c, r) = (t(x0+c, y0+r), t(x0+c+1, y0+r) - t(x0+c, y0+r)), zero border.  A warp stages
    // rows of a slice: each texel is loaded once, its right neighbour comes from the next lane.
    const int lane = threadIdx.x & 31;
    {
        constexpr int kCols = T / 32 + 1;  // lanes cover columns 0 .. T
        const int rows = ty + 1;
        constexpr int kUnroll = kThr == 384 ? 2 : C::Large ? 8 : 4;  // rows in flight (small tiles of one slice: 40 registers)
#pragma unroll kUnroll
        for (int q = threadIdx.x >> 5; q < S * rows; q += kThr / 32) {
            const int z = S == 1 ? 0 : q / rows, r = q - z * rows;
            const int gy = y0 + r;
            const bool rv = (unsigned)gy < (unsigned)g.ny;
            const float *row = image(z) + ((long long)gy * g.nx + x0);
            float t[kCols + 1];
#pragma unroll
            for (int u = 0; u < kCols; ++u) {
                const int c = lane + 32 * u;
                t[u] = (rv && (unsigned)(x0 + c) < (unsigned)g.nx) ? row[c] : 0.0f;
            }
            t[kCols] = 0.0f;
            unsigned char *dst = smem_raw + (size_t)z * C::Plane + (size_t)(r * C::P + lane) * 8;
#pragma unroll
            for (int u = 0; u < kCols; ++u) {
                const float a = __shfl_down_sync(0xffffffffu, t[u], 1), b = __shfl_sync(0xffffffffu, t[u + 1], 0);
                const float t1 = lane == 31 ? b : a;
                if (lane + 32 * u < T) *reinterpret_cast<float2 *>(dst + 256 * u) = make_float2(t[u], t1 - t[u]);
            }
        }
    }
    // owned base-texel ranges (the union over tiles is [-1, n-1])
    const float xlo = (float)x0, xhi = (float)min(x0 + tx, g.nx);
    const float ylo = (float)y0, yhi = (float)min(y0 + ty, g.ny);
    for (int k = threadIdx.x; k < kn; k += kThr) {
        const float2 cs = trig[sub + (k0 + k) * step];
        s_cs[k] = make_float4(cs.x, cs.y, 1.0f / cs.x, 1.0f / cs.y);
        // rays that can reach the tile: its corners on the detector axis, X = (x - nx/2) c -
        // (y - ny/2) s + cx (rounding stays far below the 0.25 allowed on either side)
        float pmin = 3.0e38f, pmax = -3.0e38f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float p = (((q & 1) ? xhi : xlo) - g.hx) * cs.x - (((q & 2) ? yhi : ylo) - g.hy) * cs.y + g.cx;
            pmin = fminf(pmin, p);
            pmax = fmaxf(pmax, p);
        }
        const int xa = max(0, (int)ceilf(pmin - 0.25f)), xb = min(g.px - 1, (int)floorf(pmax + 0.25f));
        s_ray[k] = make_int4(xa, xb, 0, xb < xa ? 0 : (xb - xa) / kRaysPerWarp + 1);
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // the angles' item ranges: a running sum of their ray groups (warp 0)
        int carry = 0;
        for (int b = 0; b < kn; b += 32) {
            const int k = b + lane;
            const int n = k < kn ? s_ray[k].w : 0;
            int v = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += t;
            }
            if (k < kn) {
                s_ray[k].z = carry + v - n;
                s_ray[k].w = carry + v;
            }
            carry += __shfl_sync(0xffffffffu, v, 31);
        }
    }
    __syncthreads();

    const int D = g.depth;
    const int total = s_ray[kn - 1].w;
    // shared address of element (col, row) from the round-down bits of the coordinates, the biases
    // folded into base2 (mod 2^32): bits(1.5*2^24 + 2j) = kBias24 + j
    const unsigned sbase = (unsigned)__cvta_generic_to_shared(smem_raw);
    constexpr unsigned kRow = C::P * 8, kBias24 = 0x4BC00000u;
    const unsigned base2 = sbase - kBias24 * (2u * kRow) - (unsigned)y0 * kRow - ((unsigned)XCT_FLOOR_BIAS + (unsigned)x0) * 8u;
    const f2x M23 = f2_pack(kMagic, kMagic), M24 = f2_pack(2.0f * kMagic, 2.0f * kMagic), one2 = f2_pack(1.0f, 1.0f);
    const f2x step2 = f2_pack(8.0f, 8.0f);
    const unsigned alo = sbase, ahi = sbase + C::Plane - 8;
    const int ray = lane / kLanesPerRay;  // ray within the warp's 8
    const int ph = lane % kLanesPerRay;   // sample phase of this lane
    // lane phase 0/1 bound the x coordinate, 2/3 the y coordinate (lower / upper Y limit)
    const bool bound_x = ph < 2;
    const bool upper = (ph & 1) != 0;
    const float blo = bound_x ? xlo : ylo, bhi = bound_x ? xhi : yhi;
    double *accl = accum(S > 1 && ph < S ? ph : 0);

    // items (angle, 8 consecutive rays), strided over the warps
    int k = 0;
    for (int item = threadIdx.x >> 5; item < total; item += kThr / 32) {
        int4 rr = s_ray[k];
        while (item >= rr.w) rr = s_ray[++k];
        const float4 cs = s_cs[k];
        const float c = cs.x, s = cs.y;
        const int X = rr.x + (item - rr.z) * kRaysPerWarp + ray;
        const float Xc = (float)X - g.cx;
        const float ax = fmaf(Xc, c, g.hx);
        const float ay = fmaf(Xc, -s, g.hy);
        // the four interval limits of this ray, one per lane of its group: the lower (even
        // phase) or upper (odd phase) Y limit from the x (phase 0/1) or y (2/3) coordinate
        int v = 0;
        if (X <= rr.y) {
            const float a = bound_x ? ax : ay, sl = bound_x ? s : c, isl = bound_x ? cs.w : cs.z;
            if (sl != 0.0f) {
                // sl > 0: [first(u >= lo), first(u >= hi)); sl < 0: [first(u < hi), first(u < lo))
                v = first_true(((sl > 0.0f) != upper) ? blo : bhi, a, sl, isl, g.hd, D);
            } else {  // constant coordinate: all samples or none
                v = upper ? ((a >= blo && a < bhi) ? D : 0) : 0;
            }
        }
        // lower limits (even phases) max-combined, upper ones min-combined across x and y (xor 2),
        // then exchanged within the pair of lanes (xor 1)
        const int w = __shfl_xor_sync(0xffffffffu, v, 2);
        const int m = upper ? min(v, w) : max(v, w);
        const int u = __shfl_xor_sync(0xffffffffu, m, 1);
        const int ya = upper ? u : m, len = max((upper ? m : u) - ya, 0);  // this ray's samples ya .. ya+len-1
        const f2x s2 = f2_pack(s, s), c2 = f2_pack(c, c), ax2 = f2_pack(ax, ax), ay2 = f2_pack(ay, ay);
        float sum[S];
#pragma unroll
        for (int z = 0; z < S; ++z) sum[z] = 0.0f;
        if constexpr (S == 1) {
            // one slice is bound by issue, not by the data path: every ray starts at its own first
            // sample (0.165 wavefronts per sample), which saves the warp-wide limits and the edge steps
            const float yc0 = (float)(ya + ph) - g.hd;
            f2x yc2 = f2_pack(yc0, yc0 + 4.0f);
            int n = len - ph;  // samples ya + ph, + 4, + 8, ... while n > 0
            for (; n > 4; n -= 8) {
                fwd_pair<S, T, false>(yc2, s2, c2, ax2, ay2, M23, M24, one2, base2, true, true, alo, ahi, sum);
                yc2 = f2_add(yc2, step2);
            }
            if (n > 0) fwd_pair<S, T, true>(yc2, s2, c2, ax2, ay2, M23, M24, one2, base2, true, false, alo, ahi, sum);
        } else {
            // all rays start at the warp's first sample, so that the 8 rays x 4 samples of a load stay a
            // compact patch (0.14 wavefronts per sample): a ray's lane ph takes Y = y0w + ph, + 4, + 8, ...
            // Steps of 8 samples; between the latest start and the earliest end every lane is inside its ray.
            const int y0w = __reduce_min_sync(0xffffffffu, len > 0 ? ya : 0x3fffffff);
            const int steps = (__reduce_max_sync(0xffffffffu, len > 0 ? ya + len : 0) - y0w + 7) >> 3;
            const int p0 = min((__reduce_max_sync(0xffffffffu, len > 0 ? ya : 0x3fffffff) - y0w + 7) >> 3, steps);
            const int p1 = max((__reduce_min_sync(0xffffffffu, len > 0 ? ya + len : 0) - y0w) >> 3, p0);
            const float yc0 = (float)(y0w + ph) - g.hd;
            f2x yc2 = f2_pack(yc0, yc0 + 4.0f);
            int q = y0w + ph - ya;  // this lane's sample, counted from its ray's first
            int p = 0;
            auto edge = [&](int end) {
                for (; p < end; ++p) {
                    fwd_pair<S, T, true>(yc2, s2, c2, ax2, ay2, M23, M24, one2, base2, (unsigned)q < (unsigned)len,
                                         (unsigned)(q + 4) < (unsigned)len, alo, ahi, sum);
                    yc2 = f2_add(yc2, step2);
                    q += 8;
                }
            };
            edge(p0);
            for (; p < p1; ++p) {
                fwd_pair<S, T, false>(yc2, s2, c2, ax2, ay2, M23, M24, one2, base2, true, true, alo, ahi, sum);
                yc2 = f2_add(yc2, step2);
            }
            q = y0w + ph - ya + 8 * p;
            edge(steps);
        }
        // the ray's partial sums over this tile: the 4 phases, then one atomic per slice
        float fifth = 0.0f;
        const float tot = fwd_reduce<S>(sum, ph, fifth);
        if (len > 0 && XCT_IN((long long)(k0 + k) * g.px + X, 0, (long long)nrows * g.px - 1, XCT_SITE_FWD_ACC)) {
            const size_t o = (size_t)(k0 + k) * g.px + X;
            if (ph < S) atomicAdd(accl + o, (double)tot);
            if (S == 5 && ph == 0) atomicAdd(accum(S - 1) + o, (double)fifth);
        }
    }
}

// acc: [groups * S][nrows][px] doubles.
template <int S, int T>
__global__ void __launch_bounds__(FwdTile<S, T>::Threads, FwdTile<S, T>::MinBlocks)
    fwd_tiled_kernel(const float *img, double *acc, const float2 *__restrict__ trig, KGeom g, int sub, int step, int nrows,
                     const __grid_constant__ FwdSplit f, long long units)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    xct_grid_wait();
    xct_grid_trigger();
    // the run, in shared memory: it is live across the tile's loops, where registers are short
    __shared__ long long s_at, s_end;
    auto angles = [&](long long u, int k0) { return (int)min((long long)min(nrows - k0, f.cap), s_end - u); };
    if (threadIdx.x == 0) {
        if (f.chunk > 0) {
            const int tiles = (int)(units / nrows), ch = (int)blockIdx.x / tiles, t = (int)blockIdx.x - ch * tiles;
            s_at = (long long)t * nrows + ch * f.chunk;
            s_end = s_at + min(f.chunk, nrows - ch * f.chunk);
        } else {
            s_at = f.start[blockIdx.x];
            s_end = f.start[blockIdx.x + 1];
        }
    }
    __syncthreads();
    while (s_at < s_end) {
        {
            const long long u = s_at;
            const int t = (int)(u / nrows), k0 = (int)(u - (long long)t * nrows);
            const int z = t / (f.ntx * f.nty), b = t - z * (f.ntx * f.nty), by = b / f.ntx, bx = b - by * f.ntx;
            const size_t nimg = (size_t)g.nx * g.ny, nacc = (size_t)nrows * g.px;
            const float *im = img + (size_t)z * S * nimg;
            double *ac = acc + (size_t)z * S * nacc;
            fwd_tile<S, T>(
                g, [&](int q) { return S == 1 ? im : im + (size_t)q * nimg; },
                [&](int q) { return S == 1 ? ac : ac + (size_t)q * nacc; }, trig, sub, step, nrows, -1 + bx * f.tx,
                -1 + by * f.ty, f.tx, f.ty, k0, angles(u, k0), smem_raw);
        }
        __syncthreads();  // the next tile is staged over this one
        if (threadIdx.x == 0) s_at += angles(s_at, (int)(s_at % nrows));
        __syncthreads();
    }
}

// acc -> OSEM1 ratio (meas != nullptr) or raw projection, rows th = sub + k*step; clears acc.
__global__ void fwd_finalize_kernel(double *acc, const float *meas, float *out, KGeom g, int sub, int step, int nrows)
{
    xct_grid_wait();
    xct_grid_trigger();
    const int X = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y, z = blockIdx.z;
    if (X >= g.px) return;
    double *a = acc + ((size_t)z * nrows + k) * g.px + X;
    const float p = (float)*a;
    *a = 0.0;
    const int th = sub + k * step;
    const size_t o = ((size_t)z * g.pa + th) * g.px + X;
    if (meas != nullptr) {
        const float yv = xct_measured(meas + (size_t)z * g.pa * g.px, g.px, g.pa, X, th, g.fetch);
        out[o] = xct_ratio(yv, p);
    } else {
        out[o] = p;
    }
}

// Four consecutive bins (16-byte aligned pointers): float4 / double2 accesses, each bin's arithmetic
// that of the scalar kernel.
__device__ __forceinline__ void finalize4(double *acc, const float *meas, float *out)
{
    double2 *a = reinterpret_cast<double2 *>(acc);
    const double2 a0 = a[0], a1 = a[1];
    float4 y = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (meas != nullptr) y = *reinterpret_cast<const float4 *>(meas);
    a[0] = make_double2(0.0, 0.0);
    a[1] = make_double2(0.0, 0.0);
    float4 r = make_float4((float)a0.x, (float)a0.y, (float)a1.x, (float)a1.y);
    if (meas != nullptr) r = make_float4(xct_ratio(y.x, r.x), xct_ratio(y.y, r.y), xct_ratio(y.z, r.z), xct_ratio(y.w, r.w));
    *reinterpret_cast<float4 *>(out) = r;
}

// The same for 4 consecutive bins per thread (px % 4 == 0, exact measured fetch, 16-byte
// aligned sinograms).
__global__ void __launch_bounds__(256) fwd_finalize4_kernel(double *acc, const float *meas, float *out, KGeom g, int sub,
                                                            int step, int nrows)
{
    xct_grid_wait();
    xct_grid_trigger();
    const int X = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    const int k = blockIdx.y, z = blockIdx.z;
    if (X >= g.px) return;
    const int th = sub + k * step;
    const size_t o = ((size_t)z * g.pa + th) * g.px + X;
    finalize4(acc + ((size_t)z * nrows + k) * g.px + X, meas != nullptr ? meas + o : nullptr, out + o);
}

// --------------------------------------------- backprojector, one to eight slices per tile
// For the slices of one OS-EM call (one geometry) a (pixel, angle) pair reads the same bin in
// all S slices of a group, so the bin expression is evaluated once for S gathers.  A
// CTA of 256 threads owns a 32 x 32 pixel tile of S slices and stages, per angle and
// slice, the window of the tile's bins (< 48, bounded exactly by the tile corners -- the bin coordinate is
// monotone in X and in Y -- its start rounded down to a multiple of 4) with asynchronous 16-byte copies
// (zero-filled off the detector), a chunk of angles at a time.  A thread takes 4 pixels of one row (8
// apart), a warp 8 adjacent pixels in each of 4 rows: the bins one load instruction touches
// span fewer than 32 consecutive words, so no load has a bank conflict.  Per pixel and angle:
// the reference's bin expression ((Xc*c - Yc*s) + cx) + 0.5, one address, S 4-byte loads at constant
// offsets (one per slice), packed adds over slice pairs (pixel pairs for one slice) -- in angle order,
// so each slice's sum is the same bits in every form -- and the update at the end.
// Bound: the shared-memory data path from two slices on (4 B per gather and slice), issue for one (5
// instructions, 7 operations of the FP32 pipe a gather).  The small tiles also spread one slice over the SMs:
// 2048^2 has 4096 of them, and 1024 tiles of 64 x 64 would be 1.7 waves.  100 angles of one 2048^2 slice:
// 95 us (108 with 64 x 64 tiles); three slices of 509 x 487 with 31 angles: 15 (27).
constexpr int kMsSlices = 8;  // slices per group of the slice-interleaved kernels
constexpr int kBpMsT = 32;
constexpr int kBpMsThreads = 256;
constexpr int kBpMsW = 52;      // staged bins per angle and slice (>= 31|c| + 31|s| + 3 + 3 = 49.9)
constexpr int kBpMsPix = 4;     // pixels per thread, 8 apart

template <int S>
struct BpMsShared {
    static constexpr int Chunk = S == 8 ? 24 : S == 4 ? 32 : S == 2 ? 48 : 64;  // angles per staging pass
    static constexpr unsigned SliceBytes = (unsigned)(Chunk * kBpMsW * 4);      // one slice's windows
    float win[S * Chunk * kBpMsW];  // [slice][angle][bin]
    float2 scs[Chunk];              // (c, s)
    int slo[Chunk];                 // first staged bin (a multiple of 4)
    unsigned soff[Chunk];           // byte address of slice 0's entry (bits - BIAS - lo)
};

// Slices Z .. S-1 of the bin at byte address ad.
template <int S, unsigned SliceBytes, int Z = 0>
__device__ __forceinline__ void bp_loads(unsigned ad, float (&v)[S])
{
    if constexpr (Z < S) {
        v[Z] = lds_f1_at<(int)(Z * SliceBytes)>(ad);
        bp_loads<S, SliceBytes, Z + 1>(ad, v);
    }
}

// The work of one CTA: pixel tile (bx, by) of S slices (slice z: image image(z), ratio rz + z * pa * px).
// vec: 16-byte staging copies (px a multiple of 4 and a 16-byte aligned rz).
template <int S, class Image>
__device__ __forceinline__ void bp_ms_tile(const KGeom &g, Image image, const float *rz, const float2 *__restrict__ trig,
                                           int sub, int nang, int bx, int by, float ssf, float paf, int vec,
                                           BpMsShared<S> &sh)
{
    typedef BpMsShared<S> C;
    constexpr int kAcc = S == 1 ? kBpMsPix / 2 : kBpMsPix * (S / 2);
    const size_t nprj = (size_t)g.pa * g.px;
    const int X0 = bx * kBpMsT, Y0 = by * kBpMsT;
    const int X1 = min(X0 + kBpMsT, g.nx) - 1, Y1 = min(Y0 + kBpMsT, g.ny) - 1;
    const int t = threadIdx.x;
    const int tx = t & 7, ty = t >> 3;
    // pixel i of this thread: (X0 + tx + 8i, Y0 + ty); threads past the image edge of a partial
    // tile gather for the edge pixel (inside the staged window) and write nothing
    const float Yc = (float)min(Y0 + ty, Y1) - g.hy;
    float xc[kBpMsPix];
#pragma unroll
    for (int i = 0; i < kBpMsPix; ++i) xc[i] = (float)min(X0 + tx + 8 * i, X1) - g.hx;
    f2x acc[kAcc];  // S > 1: slice pairs of each pixel, [pixel][pair]; S = 1: pixel pairs
#pragma unroll
    for (int i = 0; i < kAcc; ++i) acc[i] = 0ull;
    const f2x cxp = f2_pack(g.cx, g.cx);
    const f2x hp = f2_pack(0.5f, 0.5f);
    const f2x MM = f2_pack(kMagic, kMagic);
    const unsigned wbase = (unsigned)__cvta_generic_to_shared(sh.win);

    for (int k0 = 0; k0 < nang; k0 += C::Chunk) {
        const int kn = min(C::Chunk, nang - k0);
        __syncthreads();  // the previous chunk's gathers are done with the shared arrays
        for (int k = t; k < kn; k += kBpMsThreads) {
            const float2 cs = trig[sub + (k0 + k) * g.ss];
            sh.scs[k] = cs;
            // the bin coordinate is monotone in X and in Y: the corners bound the window
            const float xa = (float)X0 - g.hx, xb = (float)X1 - g.hx;
            const float yA = (float)Y0 - g.hy, yB = (float)Y1 - g.hy;
            const float qa = yA * cs.y, qb = yB * cs.y;
            int lo = xct_floor_bits(xct_bin_coord(xa, cs.x, qa, g.cx));
            lo = min(lo, xct_floor_bits(xct_bin_coord(xb, cs.x, qa, g.cx)));
            lo = min(lo, xct_floor_bits(xct_bin_coord(xa, cs.x, qb, g.cx)));
            lo = min(lo, xct_floor_bits(xct_bin_coord(xb, cs.x, qb, g.cx)));
            lo &= ~3;  // the bias is a multiple of 4: this rounds the bin down to one
            sh.slo[k] = lo - XCT_FLOOR_BIAS;
            // slice 0's entry for floor bits fb: wbase + 4*(k*W + fb - lo)  (mod 2^32)
            sh.soff[k] = wbase + 4u * (unsigned)(k * kBpMsW) - 4u * (unsigned)lo;
        }
        __syncthreads();
        // window (z, k) = ratio[z0 + z][th_k][lo_k .. lo_k + W), 0 off the detector
        if (vec) {
            constexpr int kQ = kBpMsW / 4;
            for (int i = t; i < kn * S * kQ; i += kBpMsThreads) {
                const int q = i % kQ, r = i / kQ;
                const int z = r % S, k = r / S;
                const int bin = sh.slo[k] + 4 * q;
                const int th = sub + (k0 + k) * g.ss;
                const float *row = rz + (size_t)z * nprj + (size_t)th * g.px;
                const int nb = bin < 0 ? 0 : min(4, g.px - bin);
                const unsigned dst = wbase + (unsigned)z * C::SliceBytes + 4u * (unsigned)(k * kBpMsW + 4 * q);
                cp_async16(dst, nb > 0 ? (const void *)(row + bin) : (const void *)row, nb > 0 ? 4u * (unsigned)nb : 0u);
            }
        } else {
            for (int i = t; i < kn * S * kBpMsW; i += kBpMsThreads) {
                const int j = i % kBpMsW, r = i / kBpMsW;
                const int z = r % S, k = r / S;
                const int bin = sh.slo[k] + j;
                const int th = sub + (k0 + k) * g.ss;
                const float *row = rz + (size_t)z * nprj + (size_t)th * g.px;
                const bool in = (unsigned)bin < (unsigned)g.px;
                const unsigned dst = wbase + (unsigned)z * C::SliceBytes + 4u * (unsigned)(k * kBpMsW + j);
                cp_async4(dst, in ? (const void *)(row + bin) : (const void *)row, in ? 4u : 0u);
            }
        }
        cp_async_wait_all();
        __syncthreads();
        const unsigned wlo = wbase, whi = wbase + 4u * (unsigned)(kn * kBpMsW - 1);
        (void)wlo;
        (void)whi;
        for (int k = 0; k < kn; ++k) {
            const float c = sh.scs[k].x, s = sh.scs[k].y;
            const unsigned off = sh.soff[k];
            const float q = Yc * s;
#pragma unroll
            for (int j = 0; j < kBpMsPix / 2; ++j) {
                // the bin expression for pixels 2j and 2j+1.  Xc*c - q in scalar: ptxas contracts a packed
                // multiply feeding a packed subtract into one fused operation whatever the rounding
                // modifiers, and the reference rounds the product and the difference separately
                const float pa_ = xc[2 * j] * c, pb_ = xc[2 * j + 1] * c;
                const f2x tt = f2_add_rd(f2_add(f2_add(f2_pack(pa_ - q, pb_ - q), cxp), hp), MM);
                int b0, b1;
                f2_unpack_bits(tt, b0, b1);
                const unsigned ad[2] = {(unsigned)b0 * 4u + off, (unsigned)b1 * 4u + off};
                float v[2][S];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    if (XCT_IN(ad[u], wlo, whi, XCT_SITE_BP_WIN)) {
                        bp_loads<S, C::SliceBytes>(ad[u], v[u]);
                    } else {
#pragma unroll
                        for (int z = 0; z < S; ++z) v[u][z] = 0.0f;
                    }
                }
                if constexpr (S == 1) {
                    acc[j] = f2_add(acc[j], f2_pack(v[0][0], v[1][0]));
                } else {
#pragma unroll
                    for (int u = 0; u < 2; ++u)
#pragma unroll
                        for (int h = 0; h < S / 2; ++h) {
                            f2x &a = acc[(2 * j + u) * (S / 2) + h];
                            a = f2_add(a, f2_pack(v[u][2 * h], v[u][2 * h + 1]));
                        }
                }
            }
        }
    }
    const int Y = Y0 + ty;
    if (Y > Y1) return;
#pragma unroll
    for (int i = 0; i < kBpMsPix; ++i) {
        const int X = X0 + tx + 8 * i;
        if (X > X1) continue;
        const size_t o = (size_t)Y * g.nx + X;
        if constexpr (S == 1) {
            float v0, v1;
            f2_unpack(acc[i / 2], v0, v1);
            float *p = image(0) + o;
            *p = xct_update(*p, i & 1 ? v1 : v0, ssf, paf);
        } else {
#pragma unroll
            for (int h = 0; h < S / 2; ++h) {
                float v0, v1;
                f2_unpack(acc[i * (S / 2) + h], v0, v1);
                float *p = image(2 * h) + o;
                *p = xct_update(*p, v0, ssf, paf);
                p = image(2 * h + 1) + o;
                *p = xct_update(*p, v1, ssf, paf);
            }
        }
    }
}

// grid: (ntx*nty tiles of 32 x 32, 1, dN / S slice groups).
template <int S>
__global__ void __launch_bounds__(kBpMsThreads) bp_ms_kernel(float *img, const float *ratio,
                                                             const float2 *__restrict__ trig, KGeom g, int sub,
                                                             int nang, int ntx, float ssf, float paf, int vec)
{
    __shared__ __align__(16) BpMsShared<S> sh;
    xct_grid_wait();
    xct_grid_trigger();
    const size_t z0 = (size_t)blockIdx.z * S, nimg = (size_t)g.nx * g.ny;
    float *im = img + z0 * nimg;
    bp_ms_tile<S>(
        g, [&](int z) { return im + (size_t)z * nimg; }, ratio + z0 * ((size_t)g.pa * g.px), trig, sub, nang,
        (int)blockIdx.x % ntx, (int)blockIdx.x / ntx, ssf, paf, vec, sh);
}

// ----------------------------------------------------------------- batched launches
// One subset step of many slices of different shapes, one launch per kernel and pack size.  Slices
// of one geometry go in packs of four and of two through the grouped forward projector and the
// several-slice backprojector, one CTA per (pack, tile) unit; the others one by one on the large tiles in the same
// way, or on smaller ones through persistent CTAs that take (slice, tile) units from a device queue (an atomic counter) until the units run
// out.  The single slices' backprojection has one CTA per unit too: what a few of them beside packs take is the
// time of one CTA over all angles, and on tiles of 64 x 64 that made packs slower than no packs (two
// geometries of three slices 300 and 320 wide, 240 and 270 angles: 663 us an iteration against 591; now 291
// against 334).  Units of pack (slice) i are [base[i], base[i+1]); they are independent within a launch, so
// there is no waiting on other CTAs.
// A pack pays per slice what the forward and backward kernels of several slices save (coordinates,
// addresses and weights once), and takes the large tiles, one CTA per SM: one iteration of 24 slices, 12
// geometries 512 to 2048 wide, takes 27.7 ms in packs of two and 39.0 one by one; 21 of seven geometries 570 to
// 1140 wide, in packs of two and single slices, 8.02 ms and 9.61; 6 of three, 200 to 400 wide, 0.32 and 0.37.
__device__ __forceinline__ int queue_take(int *queue, int *s_unit)
{
    if (threadIdx.x == 0) *s_unit = atomicAdd(queue, 1);
    __syncthreads();
    const int u = *s_unit;
    __syncthreads();
    return u;
}

// Slice owning unit u: the last i with base[i] <= u (binary search, one thread).
__device__ __forceinline__ int unit_item(const int *__restrict__ base, int n, int u, int *s_item)
{
    if (threadIdx.x == 0) {
        int lo = 0, hi = n - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (base[mid] <= u) lo = mid;
            else hi = mid - 1;
        }
        *s_item = lo;
    }
    __syncthreads();
    const int i = *s_item;
    __syncthreads();
    return i;
}

template <int T>
__global__ void __launch_bounds__(FwdTile<1, T>::Threads, FwdTile<1, T>::MinBlocks) fwd_batched_kernel(const XctItemDev *__restrict__ items,
                                                                     const int *__restrict__ base, int n, int sub,
                                                                     int *queue)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_unit, s_item;
    const int total = base[n];
    for (;;) {
        const int u = queue_take(queue, &s_unit);
        if (u >= total) break;
        const int i = unit_item(base, n, u, &s_item);
        const XctItemDev &it = items[i];
        const KGeom &g = it.g;
        const int nrows = it.cover ? (g.pa - sub + g.ss - 1) / g.ss : g.pa / g.ss;
        const int local = u - base[i];
        const int tiles = it.fwd_ntx * it.fwd_nty;
        const int t = local % tiles, ch = local / tiles;
        fwd_tile<1, T>(
            g, [&](int) { return it.img; }, [&](int) { return it.acc; }, it.trig, sub, g.ss, nrows,
            -1 + t % it.fwd_ntx * T, -1 + t / it.fwd_ntx * T, T, T, ch * g.fwd_chunk, g.fwd_chunk, smem_raw);
        __syncthreads();  // the tile in shared memory is restaged by the next unit
    }
}

// grid: one CTA per forward unit; pack i is the slices items[i * S] .. items[i * S + S - 1].
template <int S, int T>
__global__ void __launch_bounds__(FwdTile<S, T>::Threads, FwdTile<S, T>::MinBlocks)
    fwd_pack_kernel(const XctItemDev *__restrict__ items, const int *__restrict__ base, int n, int sub)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_item;
    const int u = blockIdx.x, i = unit_item(base, n, u, &s_item);
    const XctItemDev *pk = items + (size_t)i * S;
    const KGeom &g = pk->g;
    const int nrows = pk->cover ? (g.pa - sub + g.ss - 1) / g.ss : g.pa / g.ss;
    const int local = u - base[i];
    const int tiles = pk->fwd_ntx * pk->fwd_nty;
    const int t = local % tiles, ch = local / tiles;
    fwd_tile<S, T>(
        g, [&](int z) { return pk[z].img; }, [&](int z) { return pk[z].acc; }, pk->trig, sub, g.ss, nrows,
        -1 + t % pk->fwd_ntx * T, -1 + t / pk->fwd_ntx * T, T, T, ch * g.fwd_chunk, g.fwd_chunk, smem_raw);
}

// grid: one CTA per finalize unit (a ratio row of an item's largest subset), base[n] of them.  Four bins per
// thread where the row allows it, so that a row is one or two rounds of loads: bound by their latency, a bin
// at a time took 107 us per subset of 24 slices (512 to 2048 bins wide), 3.5 % of the step.
__global__ void fwd_finalize_batched_kernel(const XctItemDev *__restrict__ items, const int *__restrict__ base,
                                            int n, int sub)
{
    __shared__ int s_item;
    const int u = blockIdx.x;
    const int i = unit_item(base, n, u, &s_item);
    const XctItemDev &it = items[i];
    const KGeom &g = it.g;
    const int nrows = it.cover ? (g.pa - sub + g.ss - 1) / g.ss : g.pa / g.ss;
    const int k = u - base[i];  // one unit per ratio row of the largest subset
    if (k >= nrows) return;
    const int th = sub + k * g.ss, px = g.px, pa = g.pa, fetch = g.fetch;
    double *acc = it.acc + (size_t)k * px;
    float *out = it.ratio + (size_t)th * px;
    const float *meas = it.sino;
    if (px % 4 == 0 && fetch == XCT_FETCH_EXACT && (((size_t)acc | (size_t)out | (size_t)meas) & 15u) == 0) {
        for (int X = (int)threadIdx.x * 4; X < px; X += (int)blockDim.x * 4)
            finalize4(acc + X, meas + (size_t)th * px + X, out + X);
        return;
    }
    for (int X = threadIdx.x; X < px; X += blockDim.x) {
        const float p = (float)acc[X];
        acc[X] = 0.0;
        out[X] = xct_ratio(xct_measured(meas, px, pa, X, th, fetch), p);
    }
}

// grid: one CTA per backprojection unit; a pack's ratio images lie one after the other.
template <int S>
__global__ void __launch_bounds__(kBpMsThreads) bp_pack_kernel(const XctItemDev *__restrict__ items,
                                                               const int *__restrict__ base, int n, int sub)
{
    __shared__ __align__(16) BpMsShared<S> sh;
    __shared__ int s_item;
    const int u = blockIdx.x, i = unit_item(base, n, u, &s_item);
    const XctItemDev *pk = items + (size_t)i * S;
    const KGeom &g = pk->g;
    const int nang = (g.pa - sub + g.ss - 1) / g.ss;
    const int t = u - base[i];
    const int vec = g.px % 4 == 0 && ((size_t)pk->ratio & 15u) == 0;
    bp_ms_tile<S>(
        g, [&](int z) { return pk[z].img; }, pk->ratio, pk->trig, sub, nang, t % pk->bp_ntx, t / pk->bp_ntx, (float)g.ss,
        (float)g.pa, vec, sh);
}

}  // namespace

// ---------------------------------------------------------------- tile-size dispatch
bool xct_fwd_tile_valid(int T) { return T == 44 || T == 60 || T == 76 || T == 92; }

// Raises a kernel's dynamic shared-memory limit once per device.  Host threads may race on
// the first call of a device: the flags are atomic, and setting the attribute twice is
// harmless.  Devices beyond the table set it on every call.
static int smem_attr(const void *fn, size_t smem, std::atomic<bool> *done)
{
    int dev = 0;
    XCT_CUDA_TRY(cudaGetDevice(&dev));
    const bool cached = dev >= 0 && dev < 64;
    if (!cached || !done[dev].load(std::memory_order_acquire)) {
        XCT_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (cached) done[dev].store(true, std::memory_order_release);
    }
    return XCT_OK;
}

// Calls f(std::integral_constant<int, T>) for the plan's tile side T.
template <class F>
static int with_tile(int T, F &&f)
{
    switch (T) {
    case 44: return f(std::integral_constant<int, 44>{});
    case 60: return f(std::integral_constant<int, 60>{});
    case 76: return f(std::integral_constant<int, 76>{});
    case 92: return f(std::integral_constant<int, 92>{});
    default: return xct_fail(XCT_E_INVALID, "forward tile side must be 44, 60, 76 or 92");
    }
}

// Work units of a pack of S slices (the forward tile side and chunk are g.fwd_T and g.fwd_chunk).
void xct_batched_units(const KGeom &g, int S, int &fwd_ntx, int &fwd_nty, int &fwd_units, int &fin_units, int &bp_ntx,
                       int &bp_units)
{
    fwd_ntx = (g.nx + 1 + g.fwd_T - 1) / g.fwd_T;
    fwd_nty = (g.ny + 1 + g.fwd_T - 1) / g.fwd_T;
    const int rows = (g.pa + g.ss - 1) / g.ss;  // the largest subset (cover mode)
    fwd_units = fwd_ntx * fwd_nty * ((rows + g.fwd_chunk - 1) / g.fwd_chunk);
    fin_units = rows;
    bp_ntx = (g.nx + kBpMsT - 1) / kBpMsT;
    bp_units = bp_ntx * ((g.ny + kBpMsT - 1) / kBpMsT);
}

// Forward tile side of a pack of S slices.
int xct_pack_tile(int S) { return S == 4 ? FwdGroup<4>::Large : S == 2 ? FwdGroup<2>::Large : FwdGroup<1>::Large; }

// Persistent grid of the single slices' forward launch.
int xct_batched_grid(int sm_count, int fwd_T, int &fwd_grid)
{
    int a = 0;
    int rc = with_tile(fwd_T, [&](auto tc) -> int {
        constexpr int T = decltype(tc)::value;
        static std::atomic<bool> done[64];
        int r = smem_attr((const void *)fwd_batched_kernel<T>, FwdTile<1, T>::Smem, done);
        if (r) return r;
        XCT_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, fwd_batched_kernel<T>, FwdTile<1, T>::Threads,
                                                                   FwdTile<1, T>::Smem));
        return XCT_OK;
    });
    if (rc) return rc;
    fwd_grid = sm_count * (a > 0 ? a : 1);
    return XCT_OK;
}

template <int S>
static int launch_fwd_pack(const XctBatchStep &b, int q, int sub, cudaStream_t st)
{
    constexpr int T = FwdGroup<S>::Large;
    static std::atomic<bool> done[64];
    const int r = smem_attr((const void *)fwd_pack_kernel<S, T>, FwdTile<S, T>::Smem, done);
    if (r) return r;
    fwd_pack_kernel<S, T><<<b.fwd_units[q], FwdTile<S, T>::Threads, FwdTile<S, T>::Smem, st>>>(
        b.items + b.first(q), b.fwd_base[q], b.packs[q], sub);
    XCT_CUDA_TRY(cudaGetLastError());
    return XCT_OK;
}

// The forward launch of the single slices of one subset step (the autotuner times it alone).
int launch_fwd_batched(const XctBatchStep &b, int sub, int *queue, cudaStream_t st)
{
    if (b.large) return launch_fwd_pack<1>(b, 2, sub, st);
    return with_tile(b.fwd_T, [&](auto tc) -> int {
        constexpr int T = decltype(tc)::value;
        fwd_batched_kernel<T><<<b.fwd_grid, FwdTile<1, T>::Threads, FwdTile<1, T>::Smem, st>>>(
            b.items + b.first(2), b.fwd_base[2], b.packs[2], sub, queue);
        XCT_CUDA_TRY(cudaGetLastError());
        return XCT_OK;
    });
}

// One subset step.  The launches of the pack sizes in use run side by side (sizes beyond the first on
// side streams, so that one's last CTAs and the next one's first share the SMs).
int launch_osem_step_batched(const XctBatchStep &b, int sub, int *queue, cudaStream_t st, const XctBatchSide &side)
{
    auto parallel = [&](auto &&launch) -> int {
        int used = 0, rc = XCT_OK;
        for (int q = 0; q < 3; ++q)
            if (b.packs[q] > 0) ++used;
        if (used > 1) XCT_CUDA_TRY(cudaEventRecord(side.fork, st));
        int k = 0;
        for (int q = 0; q < 3; ++q) {
            if (b.packs[q] <= 0) continue;
            const cudaStream_t on = k == 0 ? st : side.stream[k - 1];
            if (k > 0) XCT_CUDA_TRY(cudaStreamWaitEvent(on, side.fork, 0));
            if ((rc = launch(q, on))) return rc;
            if (k > 0) XCT_CUDA_TRY(cudaEventRecord(side.join[k - 1], on));
            ++k;
        }
        for (int j = 0; j + 1 < used; ++j) XCT_CUDA_TRY(cudaStreamWaitEvent(st, side.join[j], 0));
        return XCT_OK;
    };
    int rc = parallel([&](int q, cudaStream_t on) -> int {
        return q == 0 ? launch_fwd_pack<4>(b, q, sub, on)
               : q == 1 ? launch_fwd_pack<2>(b, q, sub, on)
                        : launch_fwd_batched(b, sub, queue, on);
    });
    if (rc) return rc;
    if (b.fin_units > 0) {
        fwd_finalize_batched_kernel<<<b.fin_units, 256, 0, st>>>(b.items, b.fin_base, b.m, sub);
        XCT_CUDA_TRY(cudaGetLastError());
    }
    return parallel([&](int q, cudaStream_t on) -> int {
        const XctItemDev *it = b.items + b.first(q);
        if (q == 0)
            bp_pack_kernel<4><<<b.bp_units[q], kBpMsThreads, 0, on>>>(it, b.bp_base[q], b.packs[q], sub);
        else if (q == 1)
            bp_pack_kernel<2><<<b.bp_units[q], kBpMsThreads, 0, on>>>(it, b.bp_base[q], b.packs[q], sub);
        else
            bp_pack_kernel<1><<<b.bp_units[q], kBpMsThreads, 0, on>>>(it, b.bp_base[q], b.packs[q], sub);
        XCT_CUDA_TRY(cudaGetLastError());
        return XCT_OK;  // launches are counted when the captured graph is replayed
    });
}

int fwd_tiled_rows_cap() { return kAngChunk; }

int fwd_ms_slices() { return kMsSlices; }

// One forward launch over groups * S slices.
template <int S, int T>
static int launch_fwd_group(const KGeom &g, const float2 *trig, const float *img, double *acc, const FwdSplit &f, int groups,
                            int sub, int step, int nrows, cudaStream_t st)
{
    typedef FwdTile<S, T> C;
    static std::atomic<bool> done[64];
    const int r = smem_attr((const void *)fwd_tiled_kernel<S, T>, C::Smem, done);
    if (r) return r;
    return xct_launch(fwd_tiled_kernel<S, T>, dim3(f.ctas), C::Threads, C::Smem, st, img, acc, trig, g, sub, step, nrows, f,
                      (long long)f.ntx * f.nty * groups * nrows);
}

// A CTA per tile of side T and chunk of angles.
static void fwd_split_chunks(const KGeom &g, int T, int nrows, int chunk, int groups, FwdSplit &f)
{
    f.ntx = (g.nx + T) / T;  // base texels -1 .. n-1
    f.nty = (g.ny + T) / T;
    f.tx = f.ty = T;
    f.chunk = chunk;
    f.ctas = f.ntx * f.nty * groups * ((nrows + chunk - 1) / chunk);
    f.cap = chunk;
}

// Runs of equal modelled time for `blocks` CTAs per SM, on tiles as equal as T allows; returns that time (SM
// cycles; 0: more units than start[] can count).  A full tile and angle take `angle` cycles of an SM, the
// staging of a tile `stage`.  The work of a tile whose centre is further from the axis than half the detector
// is scaled by the share of half a turn in which that centre is projected onto it (a 2048^2 slice on 2048
// bins: 0.5 in the corners; with equal runs instead, corner CTAs finished early and the launch took 6 %
// longer).  A run takes the rest of its tile where another staging would cost more than that rest.
//
// Against a CTA per tile and chunk of angles, whose last wave is nearly empty at many sizes (three slices of
// 509 x 487: 64 tiles x 5 chunks on 304 places), a subset step takes, chunks / runs, with the large tiles: one slice
// of 2048^2 x 100 angles 464 / 419 us, of 512^2 x 36 28.5 / 25.5; three of 509 x 487 x 31 45.7 / 39.2; ten of 512^2 x
// 36 107 / 93.
static double fwd_split_runs(const KGeom &g, int T, int blocks, double angle, double stage, int nrows, int groups,
                             FwdSplit &f)
{
    f.ntx = (g.nx + T) / T;
    f.nty = (g.ny + T) / T;
    f.tx = (g.nx + f.ntx) / f.ntx;
    f.ty = (g.ny + f.nty) / f.nty;
    f.chunk = 0;
    f.cap = g.ms_chunk > 0 ? g.ms_chunk : kAngChunk;
    const int plane = f.ntx * f.nty;
    const long long tiles = (long long)plane * groups, units = tiles * nrows;
    if (units >= 0xffffffffLL || plane > 4096) return 0.0;
    const double fill = (double)f.tx * f.ty / ((double)T * T);
    const double one = angle * fill + 2.0 * T * (1.0 - fill);
    stage = stage * fill + 0.25 * one;  // and the last round of its rays, which fill the warps unevenly
    float weight[4096];
    double sum = 0.0, heaviest = 0.0;
    for (int t = 0; t < plane; ++t) {
        const double x = (t % f.ntx + 0.5) * f.tx - 0.5 - g.hx, y = (t / f.ntx + 0.5) * f.ty - 0.5 - g.hy;
        const double r = sqrt(x * x + y * y), h = 0.5 * g.px;
        weight[t] = (float)(r <= h ? one : one * 0.6366197723675814 * asin(h / r));
        sum += weight[t];
        heaviest = std::max(heaviest, (double)weight[t]);
    }
    const int most = (int)std::min<long long>(std::min(device_sm_count() * blocks, kMaxRuns), units);
    double left = sum * groups * nrows, longest = 0.0;  // angle work not assigned yet
    long long t = 0;
    int k = 0, i = 0;
    for (; i < most && t < tiles; ++i) {
        f.start[i] = (unsigned)(t * nrows + k);
        const long long rest = most - i, todo = tiles - t;
        const double budget = left / rest + stage * (todo > rest ? 1.0 + (double)todo / rest : 1.0);
        double used = 0.0;
        while (t < tiles) {
            const double w = weight[t % plane];
            if (used > 0.0 && i + 1 < most && budget - used < stage + w) break;
            used += stage;
            int n = nrows - k;
            if (i + 1 < most) {
                const int fit = std::max(1, (int)ceil((budget - used) / w - 0.05));
                if (fit < n && (n - fit) * w > 0.5 * stage) n = fit;
            }
            used += n * w;
            left -= n * w;
            k += n;
            if (k < nrows) break;
            k = 0;
            ++t;
        }
        longest = std::max(longest, used);
    }
    if (tiles <= most) {  // or the same number of runs for every tile, none of which crosses a boundary
        const int m = (int)std::min<long long>(most / tiles, nrows);
        const double own = (nrows + m - 1) / m * heaviest + stage;
        if (own < longest) {
            longest = own;
            i = (int)tiles * m;
            for (int q = 0; q < i; ++q) f.start[q] = (unsigned)(q / m * nrows + (long long)nrows * (q % m) / m);
        }
    }
    f.ctas = i;
    f.start[i] = (unsigned)units;
    return longest * blocks;
}

// Cycles of an SM that a full tile of S = 1 .. 5 slices and an angle take, and the tile's staging: large and
// small tiles (fits of launches on 256^2 to 2048^2 slices).
struct FwdForm {
    double angle[2], stage[2];
};
static const FwdForm kFwdForm[5] = {{{5450, 2900}, {8500, 3500}},
                                    {{3900, 2300}, {9200, 4800}},
                                    {{3700, 2060}, {9100, 5300}},
                                    {{3880, 1990}, {10700, 5600}},
                                    {{4150, 1990}, {10600, 5700}}};

// Modelled forward work of one pack of S slices in chunks of angles, and half a CTA's own time (tail).
double xct_pack_work(int nx, int ny, int S, int nrows, int chunk, double &tail)
{
    const double angle = kFwdForm[S - 1].angle[0], stage = kFwdForm[S - 1].stage[0];
    const int T = xct_pack_tile(S), n = (nrows + chunk - 1) / chunk;
    tail = 0.5 * (stage + chunk * angle);
    return (double)((nx + T) / T) * ((ny + T) / T) * n * stage + (nx + 1.0) * (ny + 1.0) / ((double)T * T) * nrows * angle;
}

// Modelled time (SM cycles) of a forward launch of `groups` groups of S slices with tile side T and
// nrows angles in chunks: the work of all tiles over the SMs, plus half a CTA's own time for the
// unevenness of the last wave.  A tile and angle take T^2 (0.15 + 0.085 S) + 7 T cycles and its
// staging 0.2 S T^2 + 400 (fits of measured launches: 2600 cycles per angle for S = 1, T = 92; 2790 for
// S = 2, T = 83; 2010 for S = 4, T = 58).
double xct_fwd_cost(int nx, int ny, int S, int T, int nrows, int chunk, int groups, int sms)
{
    double tail = 0.0;
    const double work = xct_fwd_work(nx, ny, S, T, nrows, chunk, groups, tail);
    return work / sms + tail;
}

// The two parts of it: the work of all tiles, and half a CTA's own time (tail).
double xct_fwd_work(int nx, int ny, int S, int T, int nrows, int chunk, int groups, double &tail)
{
    const double t2 = (double)T * T;
    const double angle = t2 * (0.15 + 0.085 * S) + 7.0 * T, stage = 0.2 * S * t2 + 400.0;
    const int blocks = S > 1 ? 2 : T <= 76 ? 4 : 3;
    const double area = (nx + 1.0) * (ny + 1.0) / t2 * groups;
    const double tiles = (double)((nx + T) / T) * ((ny + T) / T) * groups;
    const int n = (nrows + chunk - 1) / chunk;
    tail = 0.5 * blocks * (stage + chunk * angle);
    return tiles * n * stage + area * nrows * angle;
}

// The division of a launch over groups of S slices: the form (tile side) of least modelled time; returns whether
// that is the large one's.
template <int S>
static bool fwd_split(const KGeom &g, int nrows, int groups, FwdSplit &f)
{
    constexpr int T1 = FwdGroup<S>::Large, T2 = FwdGroup<S>::T;
    const FwdForm &m = kFwdForm[S - 1];
    FwdSplit f2;
    const double t1 = fwd_split_runs(g, T1, FwdTile<S, T1>::MinBlocks, m.angle[0], m.stage[0], nrows, groups, f);
    const double t2 = fwd_split_runs(g, T2, FwdTile<S, T2>::MinBlocks, m.angle[1], m.stage[1], nrows, groups, f2);
    if (t1 <= 0.0) fwd_split_chunks(g, T1, nrows, std::min(nrows, kAngChunk), groups, f);
    if (t1 <= 0.0 || t2 <= 0.0 || t1 <= t2) return true;
    f = f2;
    return false;
}

// Groups of S slices.  The division depends on the geometry, the angles, the groups and the cap alone, and finding
// it takes the host 5 us for a small slice and 20 for ten slices of 1024^2, so the geometry's owner keeps it: a
// call of the forward projection takes the host 12.5 us for one 192^2 slice and 17.6 for ten of 1024^2 (17.5 and
// 35 when each divided anew; 10.1 for one with its tile set by hand).
template <int S>
static int launch_fwd_groups(const KGeom &g, const float2 *trig, const float *&img, double *&acc, int &dN, int groups,
                             int sub, int step, int nrows, cudaStream_t st)
{
    if (groups <= 0) return XCT_OK;
    constexpr int T1 = FwdGroup<S>::Large, T2 = FwdGroup<S>::T;
    XctFwdSplits::Entry e;
    if (g.splits != nullptr) {
        std::lock_guard<std::mutex> lock(g.splits->mu);
        for (const XctFwdSplits::Entry &k : g.splits->kept)
            if (k.S == S && k.groups == groups && k.nrows == nrows && k.cap == g.ms_chunk) {
                e = k;
                break;
            }
    }
    if (e.S == 0) {
        e.S = S;
        e.groups = groups;
        e.nrows = nrows;
        e.cap = g.ms_chunk;
        e.large = fwd_split<S>(g, nrows, groups, e.f);
        if (g.splits != nullptr) {
            std::lock_guard<std::mutex> lock(g.splits->mu);
            g.splits->kept[g.splits->next] = e;
            g.splits->next = (g.splits->next + 1) % XctFwdSplits::kKept;
        }
    }
    const int rc = e.large ? launch_fwd_group<S, T1>(g, trig, img, acc, e.f, groups, sub, step, nrows, st)
                           : launch_fwd_group<S, T2>(g, trig, img, acc, e.f, groups, sub, step, nrows, st);
    img += (size_t)groups * S * g.nx * g.ny;
    acc += (size_t)groups * S * nrows * g.px;
    dN -= groups * S;
    return rc;
}

// Whether the launches of dN slices are bound by latency: one launch of groups of five then serves ten slices
// better than groups of four and two, and one stream better than two halves (ten slices of 256^2 x 18 angles,
// 11.8 M samples: 25.1 us a subset step, 27.1 in fours and twos, 30.6 in two halves; of 512^2 x 36, 94 M: 103
// against 96 and 97).
bool fwd_is_small(const KGeom &g, int dN, int nrows) { return (long long)g.nx * g.ny * nrows * dN <= 30000000; }

// The forward projection of dN slices into the accumulator: groups of four slices, the rest as one
// group of five, three, two or one (small batches of five, ten ...: fives); with grouping off or a tuned tile and one
// slice, every slice by itself in chunks of angles.  A tile set by hand serves every slice but, with the eight-slice
// forms on, whole groups of eight.
int launch_fwd_tiled_main(const KGeom &g, const float2 *trig, const float *img, double *acc, int dN, int sub, int step,
                          int nrows, cudaStream_t st)
{
    if (nrows <= 0 || dN <= 0) return XCT_OK;
    int rc = XCT_OK;
    if (g.fwd_group && !g.fwd_hand && (dN >= 2 || !g.fwd_tuned)) {
        if (dN % 5 == 0 && fwd_is_small(g, dN, nrows)) return launch_fwd_groups<5>(g, trig, img, acc, dN, dN / 5, sub, step, nrows, st);
        const bool five = dN > 1 && dN % 4 == 1;
        rc = launch_fwd_groups<4>(g, trig, img, acc, dN, five ? dN / 4 - 1 : dN / 4, sub, step, nrows, st);
        if (!rc && five) rc = launch_fwd_groups<5>(g, trig, img, acc, dN, 1, sub, step, nrows, st);
        if (!rc && dN == 3) rc = launch_fwd_groups<3>(g, trig, img, acc, dN, 1, sub, step, nrows, st);
        if (!rc && dN == 2) rc = launch_fwd_groups<2>(g, trig, img, acc, dN, 1, sub, step, nrows, st);
        if (!rc && dN == 1) rc = launch_fwd_groups<1>(g, trig, img, acc, dN, 1, sub, step, nrows, st);
        return rc;
    }
    if (g.fwd_group && g.fwd_hand && g.ms_chunk > 0) {
        rc = launch_fwd_groups<4>(g, trig, img, acc, dN, dN / kMsSlices * 2, sub, step, nrows, st);
        if (rc || dN == 0) return rc;
    }
    if (g.fwd_chunk <= 0 || g.fwd_chunk > kAngChunk) return xct_fail(XCT_E_INVALID, "forward angle chunk out of range");
    return with_tile(g.fwd_T, [&](auto tc) -> int {
        constexpr int T = decltype(tc)::value;
        FwdSplit f;
        fwd_split_chunks(g, T, nrows, g.fwd_chunk, dN, f);
        return launch_fwd_group<1, T>(g, trig, img, acc, f, dN, sub, step, nrows, st);
    });
}

int launch_fwd_finalize(const KGeom &g, const float *meas, float *out, double *acc, int dN, int sub, int step,
                        int nrows, cudaStream_t st)
{
    if (nrows <= 0 || dN <= 0) return XCT_OK;
    const bool vec = g.px % 4 == 0 && g.fetch == XCT_FETCH_EXACT && (((uintptr_t)meas | (uintptr_t)out) & 15u) == 0 &&
                     ((uintptr_t)acc & 15u) == 0;
    int rc = XCT_OK;
    for (int z = 0; z < dN && !rc; z += kMaxGridZ) {
        const int n = std::min(dN - z, kMaxGridZ);
        const size_t nprj = (size_t)g.pa * g.px;
        double *a = acc + (size_t)z * nrows * g.px;
        const float *m = meas != nullptr ? meas + z * nprj : nullptr;
        float *o = out + z * nprj;
        if (vec)
            rc = xct_launch(fwd_finalize4_kernel, dim3((g.px / 4 + 255) / 256, nrows, n), 256, 0, st, a, m, o, g, sub, step,
                            nrows);
        else
            rc = xct_launch(fwd_finalize_kernel, dim3((g.px + 127) / 128, nrows, n), 128, 0, st, a, m, o, g, sub, step, nrows);
    }
    return rc;
}

int launch_fwd_tiled(const KGeom &g, const float2 *trig, const float *img, const float *meas, float *out,
                     double *acc, int dN, int sub, int step, int nrows, cudaStream_t st)
{
    if (fwd_is_direct(g, dN, nrows)) return launch_fwd_direct(g, trig, img, meas, out, dN, sub, step, nrows, st);
    int rc = launch_fwd_tiled_main(g, trig, img, acc, dN, sub, step, nrows, st);
    if (rc) return rc;
    return launch_fwd_finalize(g, meas, out, acc, dN, sub, step, nrows, st);
}

// SM count of the current device, cached per device (152 if it cannot be read).
int device_sm_count()
{
    static std::atomic<int> cache[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 152;
    int v = cache[dev].load(std::memory_order_relaxed);
    if (v == 0) {
        int n = 0;
        v = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0 ? n : 152;
        cache[dev].store(v, std::memory_order_relaxed);
    }
    return v;
}

int launch_bp_update_tiled(const KGeom &g, const float2 *trig, float *img, const float *ratio, int dN, int sub,
                           cudaStream_t st)
{
    if (dN <= 0) return XCT_OK;
    if (bp_is_direct(g, dN)) return launch_bp_update_direct(g, trig, img, ratio, dN, sub, st);
    const int nang = (g.pa - sub + g.ss - 1) / g.ss;  // OSEM2's angle loop (OSEM.cl:93)
    // Slices go in eights (with the slice-interleaved kernels on), fours and pairs (with grouping on), the rest one by
    // one -- the larger forms cost less per slice, but only where their grid still gives every SM four CTAs: a subset
    // step of 16 slices of 512^2 x 48 angles, in two halves of 256 tiles, takes 194 us in eights and 159 in pairs;
    // of 768^2 (576 tiles) 322 in eights, 315 in fours; of 1024^2 (1024) 542 and 540.  Eights set by hand hold
    // whatever the size.
    const int mtx = (g.nx + kBpMsT - 1) / kBpMsT, mty = (g.ny + kBpMsT - 1) / kBpMsT;
    const int vec = g.px % 4 == 0 && ((uintptr_t)ratio & 15u) == 0;
    const long long tiles = (long long)mtx * mty, fill = 4LL * device_sm_count();
    auto run = [&](auto sc, int groups) -> int {
        constexpr int S = decltype(sc)::value;
        int rc = XCT_OK;
        for (int n; groups > 0 && !rc; groups -= n) {
            n = std::min(groups, kMaxGridZ);
            rc = xct_launch(bp_ms_kernel<S>, dim3(mtx * mty, 1, n), kBpMsThreads, 0, st, img, ratio, trig, g, sub, nang, mtx,
                            (float)g.ss, (float)g.pa, vec);
            img += (size_t)n * S * g.nx * g.ny;
            ratio += (size_t)n * S * g.pa * g.px;
            dN -= n * S;
        }
        return rc;
    };
    int rc = XCT_OK;
    if (g.ms_chunk > 0 && dN >= kMsSlices && (g.ms_hand || tiles * (dN / kMsSlices) >= fill))
        rc = run(std::integral_constant<int, 8>{}, dN / kMsSlices);
    if (!rc && g.fwd_group && dN >= 4 && tiles * (dN / 4) >= fill) rc = run(std::integral_constant<int, 4>{}, dN / 4);
    if (!rc && g.fwd_group && dN >= 2 && tiles * (dN / 2) >= fill) rc = run(std::integral_constant<int, 2>{}, dN / 2);
    if (!rc && dN >= 1) rc = run(std::integral_constant<int, 1>{}, dN);
    return rc;
}

XCT_CHECK_READER(xct_check_read_tiled)
