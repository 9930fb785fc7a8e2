// xct_adj.cu -- the exact adjoint of the forward projector.
//
// A^T: img[t] = sum over samples of w_t(sample) * sino[th][X], with the bilinear weights of the
// sample's 2x2 footprint -- the samples and weights of the forward projector (reconstShare.cl:213-241).
// The reference has no such kernel (its backProjection is a nearest-bin rule, :245-275); the
// differentiable pair and the gradient step of FISTA (FISTA.cl:211-246) use it.
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "xct_async.cuh"
#include "xct_check.cuh"
#include "xct_device.cuh"
#include "xct_f32x2.cuh"
#include "xct_ray.cuh"

namespace {

constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
constexpr int kLanesPerRay = 4, kRaysPerWarp = 32 / kLanesPerRay;

// ------------------------------------------------------------------- scatter form
// A CTA owns a T x T texel tile of S slices.  It visits every sample whose base texel lies in
// [x0-1, x0+T) x [y0-1, y0+T) (exactly those whose footprint touches the tile), scatters its four
// weighted values into shared accumulators and writes its own T x T texels once -- no global
// atomics, no overlap between tiles.
//
// Accumulation.  Shared-memory integer atomics run at the rate of loads, whatever number of lanes
// name the same word; float ones loop (47 cycles a warp instruction without, 1500 with such
// collisions).  So the contributions of a window of kAdjWin angles are scattered as 32-bit
// fixed-point integers, with a power-of-two scale from the window's largest |ray value| vmax < 2^e: every
// contribution is at most 2^22 units and converts with one add of 1.5*2^23 (its low bits hold the
// rounded value), and no texel can overflow: it receives at most six taps per angle (the half-open
// 2x2 cell around it holds at most five samples of the rotated unit lattice, one more allowed for
// coordinate rounding), 192 * 2^22 < 2^30 per window.  A ray's scale follows its own size: rays of at
// least vmax * 2^-6 use level 0 (unit 2^(e-22)), of at least vmax * 2^-12 level 1, of at least
// vmax * 2^-18 level 2, each level its own accumulators and a unit 2^6 finer -- so every
// contribution rounds by at most 2^-16 of its ray's value (below the weight error of float32 sample
// coordinates) and the lanes of a warp stay in step.  (A ray below vmax * 2^-18, and every ray of a
// window with a non-finite value or one above 1e30, scatters float atomics.  With one level, 4 %
// of normally distributed rays took that path, and a 1024^2 x 720-angle adjoint 2.86 ms; now 1.0.)
// After the window every thread adds its texels' integers, unscaled, to the float totals, so the
// result does not depend on the order of the atomics.
//
// Bank conflicts.  An integer atomic is served one lane per bank and wavefront, lanes that name the same
// word included.  8 rays x 4 consecutive samples per warp at the pitches below take 2.5 (T = 64) to 2.9
// wavefronts per atomic of 32 samples (a CPU model over angles and pitches; 3.3 at pitch 34 for T = 32,
// and 4.2 measured when the atomics were ordered by the parity of rows and columns, which suits loads
// but makes neighbouring samples name the same word).
//
// Bound: issue (about 28 instructions per sample, four of them atomics), then the atomics' data path.
constexpr int kAdjWin = 32;

template <int S, int T>
struct AdjTile {
    static constexpr int R = T + 2;  // texel rows and columns x0-1 .. x0+T, y0-1 .. y0+T
    static constexpr int P = T == 16 ? 20 : T == 32 ? 44 : T == 44 ? 52 : 76;
    static constexpr int Slice = P * R;  // words
    static constexpr int Threads = T == 32 ? 256 : 512;
    static constexpr size_t Sums = (size_t)S * Slice * 4;      // float totals
    static constexpr size_t TableOff = (4 * Sums + 15) & ~(size_t)15;  // after the integers [S][3 levels][Slice]
    static constexpr size_t Smem = TableOff + kAdjWin * 32 + 2 * S * sizeof(int);
    static_assert(P >= R, "tile pitch");
};

__device__ __forceinline__ void red_add(unsigned addr, int v)
{
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void red_add_f(unsigned addr, float v)
{
    asm volatile("red.shared.add.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((e + 127) << 23); }  // -126 <= e <= 127

// grid: (ntx*nty tiles, 1, groups of S slices).  The angles are th = sub + k*step for k < nang; with base
// non-null the output is base + scale_out * (A^T sino) (a gradient step).
template <int S, int T>
__global__ void __launch_bounds__(AdjTile<S, T>::Threads, 1024 / AdjTile<S, T>::Threads) adj_scatter_kernel(const float *__restrict__ sino,
                                                                             float *__restrict__ img,
                                                                             const float2 *__restrict__ trig, KGeom g,
                                                                             int ntx, int sub, int step, int nang,
                                                                             const float *__restrict__ base, float scale_out)
{
    typedef AdjTile<S, T> C;
    constexpr int kThr = C::Threads, kWarps = kThr / 32;
    constexpr unsigned kRow = C::P * 4, kSl = C::Slice * 4;  // bytes
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float *sums = reinterpret_cast<float *>(smem_raw);
    int *ints = reinterpret_cast<int *>(smem_raw + C::Sums);
    float4 *s_cs = reinterpret_cast<float4 *>(smem_raw + C::TableOff);
    int4 *s_ray = reinterpret_cast<int4 *>(s_cs + kAdjWin);
    unsigned *s_max = reinterpret_cast<unsigned *>(s_ray + kAdjWin);  // two windows' largest |value| bits per slice
    const int bx = (int)blockIdx.x % ntx, by = (int)blockIdx.x / ntx;
    const int z0 = (int)blockIdx.z * S;
    const size_t nprj = (size_t)g.pa * g.px, nimg = (size_t)g.nx * g.ny;
    const int x0 = bx * T, y0 = by * T;  // owned texels [x0, x0+T) x [y0, y0+T)
    for (int i = threadIdx.x; i < 4 * S * C::Slice; i += kThr) sums[i] = 0.0f;  // and the integers
    if (threadIdx.x < 2 * S) s_max[threadIdx.x] = 0u;
    const float *sn = sino + (size_t)z0 * nprj;
    // base texels whose footprint touches the tile
    const float xlo = (float)(x0 - 1), xhi = (float)min(x0 + T, g.nx);
    const float ylo = (float)(y0 - 1), yhi = (float)min(y0 + T, g.ny);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int D = g.depth;
    const int ray = lane / kLanesPerRay, ph = lane % kLanesPerRay;
    const bool bound_x = ph < 2, upper = (ph & 1) != 0;
    const float blo = bound_x ? xlo : ylo, bhi = bound_x ? xhi : yhi;
    // byte offset of texel (x, y) from the floor bits (x + BIAS, ...), biases folded in (mod 2^32)
    constexpr unsigned kBias = (unsigned)XCT_FLOOR_BIAS;
    const unsigned sints = (unsigned)__cvta_generic_to_shared(ints), ssums = (unsigned)__cvta_generic_to_shared(sums);
    const unsigned base0 = (1u - (unsigned)y0 - kBias) * kRow + (1u - (unsigned)x0 - kBias) * 4u;
    const f2x M23 = f2_pack(kMagic, kMagic), one2 = f2_pack(1.0f, 1.0f), step2 = f2_pack(8.0f, 8.0f);

    for (int w0 = 0, win = 0; w0 < nang; w0 += kAdjWin, win ^= 1) {
        const int kn = min(kAdjWin, nang - w0);
        if (warp == 0) {
            // lane k: angle w0 + k, the rays that can reach the tile (its corners on the detector axis;
            // rounding stays far below the 0.25 allowed), and the running sum of their groups of eight
            int xa = 0, n = 0, xb = -1;
            if (lane < kn) {
                const float2 cs = __ldg(trig + sub + (w0 + lane) * step);
                s_cs[lane] = make_float4(cs.x, cs.y, 1.0f / cs.x, 1.0f / cs.y);
                float pmin = 3.0e38f, pmax = -3.0e38f;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float p = (((q & 1) ? xhi : xlo) - g.hx) * cs.x - (((q & 2) ? yhi : ylo) - g.hy) * cs.y + g.cx;
                    pmin = fminf(pmin, p);
                    pmax = fmaxf(pmax, p);
                }
                xa = max(0, (int)ceilf(pmin - 0.25f));
                xb = min(g.px - 1, (int)floorf(pmax + 0.25f));
                n = xb < xa ? 0 : (xb - xa) / kRaysPerWarp + 1;
            }
            int v = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += t;
            }
            if (lane < kn) s_ray[lane] = make_int4(xa, xb, v - n, v);
        }
        __syncthreads();  // the table; the last window's integers are cleared
        // each slice's largest |ray value| over the window, as bits: those of a NaN or an infinity are
        // above every finite value's
        for (int k = warp; k < kn; k += kWarps) {
            const int4 rr = s_ray[k];
            const float *row = sn + (size_t)(sub + (w0 + k) * step) * g.px;
            unsigned m[S];
#pragma unroll
            for (int z = 0; z < S; ++z) m[z] = 0u;
            for (int X = rr.x + lane; X <= rr.y; X += 32)
#pragma unroll
                for (int z = 0; z < S; ++z) m[z] = max(m[z], __float_as_uint(__ldg(row + z * nprj + X)) & 0x7fffffffu);
#pragma unroll
            for (int z = 0; z < S; ++z) {
                const unsigned r = __reduce_max_sync(0xffffffffu, m[z]);
                if (lane == 0) atomicMax(s_max + win * S + z, r);
            }
        }
        __syncthreads();
        if (threadIdx.x < S) s_max[(win ^ 1) * S + threadIdx.x] = 0u;  // for the next window
        float vmax[S];
        int ex[S];  // vmax < 2^ex
        bool fixed[S];
#pragma unroll
        for (int z = 0; z < S; ++z) {
            const unsigned b = s_max[win * S + z];
            vmax[z] = __uint_as_float(b);
            fixed[z] = vmax[z] < 1.0e30f && b != 0u;  // false for NaN, inf and finite windows above 1e30
            ex[z] = max((int)(b >> 23) - 126, -78);   // scales stay <= 2^112
        }
        const int total = s_ray[kn - 1].w;
        int k = 0;
        for (int item = warp; item < total; item += kWarps) {
            int4 rr = s_ray[k];
            while (item >= rr.w) rr = s_ray[++k];
            const float4 cs = s_cs[k];
            const float c = cs.x, s = cs.y;
            const int X = rr.x + (item - rr.z) * kRaysPerWarp + ray;
            const bool live = X <= rr.y;
            const float *vp = sn + (size_t)(sub + (w0 + k) * step) * g.px + X;
            // each slice's ray value: its level's scale and accumulators, or the float path
            float v[S], vs[S];
            unsigned lv[S], flt = 0;
            bool any = false;
#pragma unroll
            for (int z = 0; z < S; ++z) {
                v[z] = live ? __ldg(vp + z * nprj) : 0.0f;
                any |= v[z] != 0.0f;
                const float a = fabsf(v[z]);
                const int l = a >= vmax[z] * 0x1p-6f ? 0 : a >= vmax[z] * 0x1p-12f ? 1 : 2;
                vs[z] = fixed[z] ? v[z] * pow2f(22 - ex[z] + 6 * l) : 0.0f;
                lv[z] = sints + (unsigned)(3 * z + l) * kSl + base0;
                if (v[z] != 0.0f && !(fixed[z] && a >= vmax[z] * 0x1p-18f)) {
                    flt |= 1u << z;
                    vs[z] = 0.0f;
                }
            }
            const float Xc = (float)X - g.cx;
            const float ax = fmaf(Xc, c, g.hx);
            const float ay = fmaf(Xc, -s, g.hy);
            int lim = 0;
            if (live) {
                const float a = bound_x ? ax : ay, sl = bound_x ? s : c, isl = bound_x ? cs.w : cs.z;
                if (sl != 0.0f) lim = first_true(((sl > 0.0f) != upper) ? blo : bhi, a, sl, isl, g.hd, D);
                else lim = upper ? ((a >= blo && a < bhi) ? D : 0) : 0;
            }
            const int w = __shfl_xor_sync(0xffffffffu, lim, 2);
            const int m = upper ? min(lim, w) : max(lim, w);
            const int u = __shfl_xor_sync(0xffffffffu, m, 1);
            const int ya = upper ? u : m;
            int n = (live && any) ? (upper ? m : u) - ya - ph : 0;  // samples ya + ph, + 4, ... while n > 0
            const float yc0 = (float)(ya + ph) - g.hd;
            const f2x s2 = f2_pack(s, s), c2 = f2_pack(c, c), ax2 = f2_pack(ax, ax), ay2 = f2_pack(ay, ay);
            f2x yc2 = f2_pack(yc0, yc0 + 4.0f);
            for (; n > 0; n -= 8) {
                // two samples: floors as round-down adds of 1.5*2^23 (the low mantissa bits), weights
                const f2x x2 = f2_fma(yc2, s2, ax2), y2 = f2_fma(yc2, c2, ay2);
                const f2x tx = f2_add_rd(x2, M23), ty = f2_add_rd(y2, M23);
                const f2x fx2 = f2_sub(x2, f2_sub(tx, M23)), fy2 = f2_sub(y2, f2_sub(ty, M23));
                const f2x gx2 = f2_sub(one2, fx2), gy2 = f2_sub(one2, fy2);
                int jx[2], jy[2];
                float fx[2], fy[2], gx[2], gy[2];
                f2_unpack_bits(tx, jx[0], jx[1]);
                f2_unpack_bits(ty, jy[0], jy[1]);
                f2_unpack(fx2, fx[0], fx[1]);
                f2_unpack(fy2, fy[0], fy[1]);
                f2_unpack(gx2, gx[0], gx[1]);
                f2_unpack(gy2, gy[0], gy[1]);
                yc2 = f2_add(yc2, step2);
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (q == 1 && n <= 4) break;
                    const unsigned o = (unsigned)jy[q] * kRow + (unsigned)jx[q] * 4u;
                    if (!XCT_IN(o + base0, 0, kSl - kRow - 8, XCT_SITE_ADJ)) continue;
#pragma unroll
                    for (int z = 0; z < S; ++z) {
                        // round(x) for |x| <= 2^22: the low bits of x + 1.5*2^23
                        const float p0 = vs[z] * gy[q], p1 = vs[z] * fy[q];
                        const unsigned b = lv[z] + o;
                        red_add(b, __float_as_int(fmaf(gx[q], p0, kMagic)) - 0x4B400000);
                        red_add(b + 4, __float_as_int(fmaf(fx[q], p0, kMagic)) - 0x4B400000);
                        red_add(b + kRow, __float_as_int(fmaf(gx[q], p1, kMagic)) - 0x4B400000);
                        red_add(b + kRow + 4, __float_as_int(fmaf(fx[q], p1, kMagic)) - 0x4B400000);
                    }
                    if (flt != 0) {
#pragma unroll
                        for (int z = 0; z < S; ++z)
                            if ((flt >> z) & 1u) {
                                const unsigned b = ssums + base0 + (unsigned)z * kSl + o;
                                red_add_f(b, gx[q] * gy[q] * v[z]);
                                red_add_f(b + 4, fx[q] * gy[q] * v[z]);
                                red_add_f(b + kRow, gx[q] * fy[q] * v[z]);
                                red_add_f(b + kRow + 4, fx[q] * fy[q] * v[z]);
                            }
                    }
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int z = 0; z < S; ++z) {
            if (!fixed[z]) continue;
            const float i0 = pow2f(ex[z] - 22), i1 = pow2f(ex[z] - 28), i2 = pow2f(ex[z] - 34);
            int *q = ints + z * 3 * C::Slice;
            for (int i = threadIdx.x; i < C::Slice; i += kThr) {
                const int q0 = q[i], q1 = q[i + C::Slice], q2 = q[i + 2 * C::Slice];
                if ((q0 | q1 | q2) != 0) {
                    sums[z * C::Slice + i] += fmaf((float)q0, i0, fmaf((float)q1, i1, (float)q2 * i2));
                    q[i] = 0;
                    q[i + C::Slice] = 0;
                    q[i + 2 * C::Slice] = 0;
                }
            }
        }
    }
    __syncthreads();
    for (int z = 0; z < S; ++z) {
        float *im = img + (size_t)(z0 + z) * nimg;
        const float *bz = base ? base + (size_t)(z0 + z) * nimg : nullptr;
        for (int i = threadIdx.x; i < T * T; i += kThr) {
            const int r = i / T, cc = i - r * T;
            const int X = x0 + cc, Y = y0 + r;
            if (X < g.nx && Y < g.ny) {
                const float a = sums[z * C::Slice + (r + 1) * C::P + cc + 1];
                const size_t o = (size_t)Y * g.nx + X;
                im[o] = bz ? fmaf(scale_out, a, __ldg(bz + o)) : a;
            }
        }
    }
}

// ------------------------------------------------------------------- gather form
// The exact adjoint over four, eight or ten slices as a gather, without atomics.  Every sample (ray X,
// index Y) of the forward projector has one base texel (floor of its coordinates); its value
// v goes to that base texel's four footprint texels with the weights gx gy, fx gy, gx fy,
// fx fy.  A thread owns one base texel (i, j) and keeps four accumulators per slice -- the
// parts its samples give to (i, j), (i+1, j), (i, j+1), (i+1, j+1) -- so each sample is
// handled by exactly one thread.  Per angle the thread finds its samples: a half-open unit
// square holds at most two points of the rotated unit sample lattice, which lie on the at
// most two rays whose lattice coordinate is within 0.717 of the square's centre, each at
// most two sample indices within 0.717 of the centre's projection on the ray; each of those
// four candidates is evaluated with the forward projector's own arithmetic (fma
// coordinates) and kept when its offset from (i, j), exact there, lies in [0, 1) in x and y --
// as integers, both halves of the offset are below the bits of 1.0 -- and its index is within
// [0, D); rays off the detector are staged as zeros.  A CTA owns 32 x BY base texels (BY = 16, or 20
// for ten slices) and writes the 31 x (BY - 1) texels whose four base texels it holds,
// texel (i, j) = A00(i, j) + A10(i-1, j) + A01(i, j-1) + A11(i-1, j-1), after staging the
// four parts in shared memory.
// The rays' values of 16 angles at a time are staged by asynchronous copies into one of two
// windows: the next chunk's copies run while this chunk is accumulated.  Most squares hold
// one sample per angle, about 9 % two and 9 % none, so a warp whose lanes each added all
// their samples at once would run two accumulation passes at almost every angle; a second
// sample instead waits in a four-slot queue per thread in shared memory
// (window address and fractions) and the queues are emptied at the end of the chunk -- about
// 1.2 passes per angle instead of 1.8.  Float sums in a fixed order given by the geometry:
// deterministic, and no fixed-point rounding.
constexpr int kAdjGBX = 32;                          // base texels per CTA row
constexpr int kAdjGW = 44;  // staged rays per angle (a 32 x 20 block needs at most 43)
constexpr int kAdjGChunk = 16;                       // angles per staging pass
template <int S>
struct AdjG {
    // base texel rows per CTA (one thread per base texel): 16 at two CTAs per SM (four and eight
    // slices), 20 at one (ten slices)
    static constexpr int BY = S <= 8 ? 16 : 20;
    static constexpr int Threads = kAdjGBX * BY;
    static constexpr unsigned QStride = 16u * Threads;  // bytes between a queue's slots
    // two windows: [slice pair][angle][ray] of float2, then the queues: [slot][thread] of
    // (window address, fx, fy); later the parts: [corner][slice][thread]; then three slots of
    // the angles' (c, -s, s, c), (c, s, -s, c) and first staged ray
    static constexpr unsigned PairBytes = (unsigned)(kAdjGChunk * kAdjGW * 8);
    static constexpr unsigned WinBytes = (unsigned)(S / 2) * PairBytes;
    static constexpr size_t CombBytes = (size_t)4 * S * Threads * 4;
    static constexpr int Queue = 4;  // queued samples per thread
    static constexpr size_t QueueBytes = (size_t)Queue * QStride;
    static constexpr size_t SlotBytes = (size_t)3 * kAdjGChunk * 36;
    static constexpr size_t Front = 2 * (size_t)WinBytes + QueueBytes;
    static constexpr size_t Smem = (Front > CombBytes ? Front : CombBytes) + SlotBytes;
};

__device__ __forceinline__ f2x lds_f2x(unsigned addr)
{
    f2x v;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(addr));
    return v;
}

// A queued sample: window address and fractions (fx, fy) in one 16-byte slot.
__device__ __forceinline__ void sts_q(unsigned addr, unsigned ad, f2x fr)
{
    asm volatile("{ .reg .b32 lo, hi; mov.b64 {lo, hi}, %2; st.shared.v4.b32 [%0], {%1, lo, hi, %1}; }"
                 :: "r"(addr), "r"(ad), "l"(fr) : "memory");
}
__device__ __forceinline__ void lds_q(unsigned addr, unsigned &ad, f2x &fr)
{
    asm volatile("{ .reg .b32 lo, hi, pad; ld.shared.v4.b32 {%0, lo, hi, pad}, [%2]; mov.b64 %1, {lo, hi}; }"
                 : "=r"(ad), "=l"(fr) : "r"(addr) : "memory");
}

// S (even) slices per CTA; the library launches S = 4 and 8 (two CTAs per SM) and 10 (one).
template <int S>
__global__ void __launch_bounds__(AdjG<S>::Threads, S <= 8 ? 2 : 1) adj_gather_kernel(const float *__restrict__ sino,
                                                                     float *__restrict__ img,
                                                                     const float2 *__restrict__ trig, KGeom g,
                                                                     int ntx, int sub, int step, int nang,
                                                                     const float *__restrict__ base, float scale_out)
{
    constexpr int P = S / 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float *part = reinterpret_cast<float *>(smem_raw);  // the window, later the parts
    float4 *scs = reinterpret_cast<float4 *>(smem_raw + AdjG<S>::Smem - AdjG<S>::SlotBytes);
    int *sxw = reinterpret_cast<int *>(scs + 6 * kAdjGChunk);
    const int tx = threadIdx.x % kAdjGBX, ty = threadIdx.x / kAdjGBX;
    const int bx = (int)blockIdx.x % ntx, by = (int)blockIdx.x / ntx;
    const int z0 = (int)blockIdx.z * S;
    const size_t nprj = (size_t)g.pa * g.px, nimg = (size_t)g.nx * g.ny;
    const float *sz = sino + (size_t)z0 * nprj;
    // base texels [bi0, bi0 + 32) x [bj0, bj0 + 16); output texels from bi0 + 1, bj0 + 1
    const int bi0 = bx * (kAdjGBX - 1) - 1, bj0 = by * (AdjG<S>::BY - 1) - 1;
    const int i = bi0 + tx, j = bj0 + ty;
    const f2x bxy = f2_pack((float)i, (float)j);
    // the square's centre, from the image's
    const float di = (float)i + 0.5f - g.hx, dj = (float)j + 0.5f - g.hy;
    const f2x di2 = f2_pack(di, di), dj2 = f2_pack(dj, dj);
    const int D = g.depth;
    const bool border = bi0 < 0 || bj0 < 0;  // holds base texels -1
    const unsigned wbase = (unsigned)__cvta_generic_to_shared(part);
    const f2x MM = f2_pack(kMagic, kMagic), M1 = f2_pack(kMagic - 1.0f, kMagic - 1.0f), one2 = f2_pack(1.0f, 1.0f);
    const f2x hxy = f2_pack(g.hx, g.hy);
    const f2x origin = f2_pack(g.cx, g.hd), first = f2_pack(g.cx - 0.717f, g.hd - 0.717f);
    f2x acc[4][P];  // [corner 00, 10, 01, 11][slice pair]
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int h = 0; h < P; ++h) acc[q][h] = 0ull;

    // one sample: fractions (fx, fy) of its base texel, window byte address ad of its ray;
    // the four bilinear weights (gx gy, fx gy, gx fy, fx fy) times the slices' ray values
    auto add = [&](unsigned ad, f2x fr, unsigned wb) {
        const f2x gr = f2_sub(one2, fr);
        float fx, fy, gx, gy;
        f2_unpack(fr, fx, fy);
        f2_unpack(gr, gx, gy);
        const float w[4] = {gx * gy, fx * gy, gx * fy, fx * fy};
        if (!XCT_IN(ad, wb, wb + AdjG<S>::WinBytes - 8, XCT_SITE_ADJ)) return;
        f2x v[P];
#pragma unroll
        for (int h = 0; h < P; ++h) v[h] = lds_f2x(ad + (unsigned)h * AdjG<S>::PairBytes);
#pragma unroll
        for (int cq = 0; cq < 4; ++cq) {
            const f2x ww = f2_pack(w[cq], w[cq]);
#pragma unroll
            for (int h = 0; h < P; ++h) acc[cq][h] = f2_fma(ww, v[h], acc[cq][h]);
        }
    };
    // this thread's queue of samples left for the end of the chunk: slot i at qb + i * stride
    const unsigned qb = wbase + 2u * AdjG<S>::WinBytes + 16u * threadIdx.x;
    int qn = 0;

    // Software pipeline over chunks of 16 angles: the rays of chunk ch + 1 are copied into the
    // other window while chunk ch is accumulated; the angles' (cos, sin) and first staged ray
    // sit in three slots (chunks ch, ch + 1, ch + 2), the (cos, sin) of chunk ch + 3 in the
    // registers of threads 0..15.
    const int nch = (nang + kAdjGChunk - 1) / kAdjGChunk;
    auto trig_of = [&](int ch) -> float2 {
        const int a = ch * kAdjGChunk + (int)threadIdx.x;
        return (ch < nch && (int)threadIdx.x < kAdjGChunk && a < nang) ? __ldg(trig + sub + a * step)
                                                                        : make_float2(0.0f, 0.0f);
    };
    auto prep = [&](int ch, float2 cs) {
        if (ch >= nch || (int)threadIdx.x >= kAdjGChunk) return;
        const int at = (ch % 3) * kAdjGChunk + (int)threadIdx.x;
        scs[2 * at] = make_float4(cs.x, -cs.y, cs.y, cs.x);
        scs[2 * at + 1] = make_float4(cs.x, cs.y, -cs.y, cs.x);
        // rays whose lattice coordinate meets the block's base squares
        float umin = 3.0e38f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float px_ = (float)(bi0 + ((q & 1) ? kAdjGBX : 0)) - g.hx;
            const float py_ = (float)(bj0 + ((q & 2) ? AdjG<S>::BY : 0)) - g.hy;
            umin = fminf(umin, px_ * cs.x - py_ * cs.y + g.cx);
        }
        sxw[at] = (int)floorf(umin) - 2;
    };
    // window (pair p, angle k, ray sxw + r) = (slice 2p, slice 2p + 1), 0 off the detector
    auto stage = [&](int ch) {
        if (ch >= nch) return;
        const int k0 = ch * kAdjGChunk, kn = min(kAdjGChunk, nang - k0), sl = (ch % 3) * kAdjGChunk;
        const unsigned wb = wbase + (unsigned)(ch & 1) * AdjG<S>::WinBytes;
        // a warp copies rows (angle, slice) of the window
        for (int q = (int)threadIdx.x >> 5; q < kn * S; q += AdjG<S>::Threads / 32) {
            const int k = q / S, z = q - k * S;
            const int X0 = sxw[sl + k];
            const float *row = sz + (size_t)z * nprj + (size_t)(sub + (k0 + k) * step) * g.px;
            const unsigned dst = wb + (unsigned)(z >> 1) * AdjG<S>::PairBytes + 8u * (unsigned)(k * kAdjGW) + 4u * (unsigned)(z & 1);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int r = ((int)threadIdx.x & 31) + 32 * u;
                if (r >= kAdjGW) break;
                const bool in = (unsigned)(X0 + r) < (unsigned)g.px;
                cp_async4(dst + 8u * (unsigned)r, in ? (const void *)(row + X0 + r) : (const void *)row, in ? 4u : 0u);
            }
        }
    };
    prep(0, trig_of(0));
    prep(1, trig_of(1));
    float2 csr = trig_of(2);
    __syncthreads();
    stage(0);
    for (int ch = 0; ch < nch; ++ch) {
        // this chunk's copies have landed; every thread is past chunk ch - 1, whose window
        // and slot are reused below
        cp_async_wait_all();
        __syncthreads();
        prep(ch + 2, csr);
        csr = trig_of(ch + 3);
        stage(ch + 1);
        const int k0 = ch * kAdjGChunk, kn = min(kAdjGChunk, nang - k0), sl = (ch % 3) * kAdjGChunk;
        const unsigned wb = wbase + (unsigned)(ch & 1) * AdjG<S>::WinBytes;
        for (int k = 0; k < kn; ++k) {
            const float4 ra = scs[2 * (sl + k)], rb = scs[2 * (sl + k) + 1];
            const f2x cs2 = f2_pack(ra.x, ra.y), sc2 = f2_pack(ra.z, ra.w);
            // the candidates: rays Xa, Xa + 1 (lattice coordinate of the cell centre - 0.717 and
            // up); on each, indices Ya, Ya + 1 (the centre's coordinate along the rays, the same on
            // every ray): the floors of both estimates, plus one
            const f2x uw = f2_fma(di2, f2_pack(rb.x, rb.y), f2_fma(dj2, f2_pack(rb.z, rb.w), first));
            const f2x tb = f2_add_rd(uw, MM);
            const f2x XY = f2_sub(tb, M1);  // (Xa, Ya) as floats
            int xb, yb;
            f2_unpack_bits(tb, xb, yb);
            const int Ya = yb - (XCT_FLOOR_BIAS - 1);
            float Xf, Yf, Xc0, Yc0;
            f2_unpack(XY, Xf, Yf);
            f2_unpack(f2_sub(XY, origin), Xc0, Yc0);  // X - cx and Y - hd, as the forward
            const float Xc1 = (Xf + 1.0f) - g.cx;
            const f2x y0 = f2_pack(Yc0, Yc0), y1 = f2_pack(Yc0 + 1.0f, Yc0 + 1.0f);  // exact: hd is a multiple of 0.5
            const f2x a0 = f2_fma(f2_pack(Xc0, Xc0), cs2, hxy), a1 = f2_fma(f2_pack(Xc1, Xc1), cs2, hxy);  // (ax, ay)
            f2x fr[4] = {f2_fma(y0, sc2, a0), f2_fma(y1, sc2, a0), f2_fma(y0, sc2, a1), f2_fma(y1, sc2, a1)};  // (x, y)
            if (border) {
                // a coordinate just below 0 belongs to base texel -1, but its offset from -1 would round to 1
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    float x, y;
                    f2_unpack(fr[q], x, y);
                    fr[q] = f2_pack(x < 0.0f ? fminf(x, -0x1p-24f) : x, y < 0.0f ? fminf(y, -0x1p-24f) : y);
                }
            }
            const bool in0 = (unsigned)Ya < (unsigned)D, in1 = (unsigned)(Ya + 1) < (unsigned)D;
            bool p[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                fr[q] = f2_sub(fr[q], bxy);
                int fxb, fyb;
                f2_unpack_bits(fr[q], fxb, fyb);
                p[q] = max((unsigned)fxb, (unsigned)fyb) < 0x3f800000u && (q & 1 ? in1 : in0);
            }
            // window address of ray Xa
            const unsigned ad = wb + 8u * (unsigned)(k * kAdjGW - sxw[sl + k] - (XCT_FLOOR_BIAS - 1)) + 8u * (unsigned)xb;
            // a unit square holds at most two samples.  The first is added now; a second one
            // (and, never seen but kept for float-rounded coordinates at the square's corners,
            // any further) waits in the queue, or is added now when the queue is full
            const bool p01 = p[0] || p[1];
            if ((p[0] && p[1]) || (p[2] && p[3]) || (p01 && (p[2] || p[3]))) {
                bool seen = p[0];
#pragma unroll
                for (int q = 1; q < 4; ++q) {
                    if (!p[q]) continue;
                    if (seen) {
                        const unsigned aq = ad + (q & 2 ? 8u : 0u);
                        if (qn < AdjG<S>::Queue) {
                            sts_q(qb + (unsigned)qn * AdjG<S>::QStride, aq, fr[q]);
                            ++qn;
                        } else {
                            add(aq, fr[q], wb);
                        }
                    }
                    seen = true;
                }
            }
            if (p01 || p[2] || p[3]) {
                const f2x f = p[0] ? fr[0] : p[1] ? fr[1] : p[2] ? fr[2] : fr[3];
                add(ad + (p01 ? 0u : 8u), f, wb);
            }
        }
        // the queued samples, while this chunk's window is still in place
        for (int i = 0; i < qn; ++i) {
            unsigned ad;
            f2x fr;
            lds_q(qb + (unsigned)i * AdjG<S>::QStride, ad, fr);
            add(ad, fr, wb);
        }
        qn = 0;
    }
    // the parts: part[corner][slice][thread]
    __syncthreads();
#pragma unroll
    for (int cq = 0; cq < 4; ++cq)
#pragma unroll
        for (int h = 0; h < P; ++h) {
            float a0, a1;
            f2_unpack(acc[cq][h], a0, a1);
            part[(cq * S + 2 * h) * AdjG<S>::Threads + threadIdx.x] = a0;
            part[(cq * S + 2 * h + 1) * AdjG<S>::Threads + threadIdx.x] = a1;
        }
    __syncthreads();
    if (tx == 0 || ty == 0 || i >= g.nx || j >= g.ny) return;
    const int t = threadIdx.x;
#pragma unroll
    for (int z = 0; z < S; ++z) {
        const float a = part[(0 * S + z) * AdjG<S>::Threads + t] + part[(1 * S + z) * AdjG<S>::Threads + t - 1] +
                        part[(2 * S + z) * AdjG<S>::Threads + t - kAdjGBX] +
                        part[(3 * S + z) * AdjG<S>::Threads + t - kAdjGBX - 1];
        const size_t o = (size_t)(z0 + z) * nimg + (size_t)j * g.nx + i;
        img[o] = base ? fmaf(scale_out, a, __ldg(base + o)) : a;
    }
}

// Launch of adj_gather_kernel<S> over `groups` groups of S slices (its shared memory opted in
// once per device).
template <int S>
static int launch_adj_gather(const KGeom &g, const float2 *trig, const float *sino, float *img, int groups, int sub,
                             int step, int nang, const float *base, float scale, cudaStream_t st)
{
    static std::atomic<bool> done[64];
    int dev = 0;
    XCT_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return xct_fail(XCT_E_INVALID, "device index out of range");
    if (!done[dev].load(std::memory_order_acquire)) {
        XCT_CUDA_TRY(cudaFuncSetAttribute((const void *)adj_gather_kernel<S>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AdjG<S>::Smem));
        done[dev].store(true, std::memory_order_release);
    }
    const int ntx = (g.nx + kAdjGBX - 2) / (kAdjGBX - 1), nty = (g.ny + AdjG<S>::BY - 2) / (AdjG<S>::BY - 1);
    adj_gather_kernel<S><<<dim3(ntx * nty, 1, groups), AdjG<S>::Threads, AdjG<S>::Smem, st>>>(sino, img, trig, g, ntx, sub,
                                                                                         step, nang, base, scale);
    g_xct_launches.fetch_add(1, std::memory_order_relaxed);
    XCT_CUDA_TRY(cudaGetLastError());
    return XCT_OK;
}

template <int S, int T>
int launch_adj_scatter(const KGeom &g, const float2 *trig, const float *sino, float *img, int groups, int sub, int step,
                       int nang, const float *base, float scale, cudaStream_t st)
{
    typedef AdjTile<S, T> C;
    static std::atomic<bool> done[64];
    int dev = 0;
    XCT_CUDA_TRY(cudaGetDevice(&dev));
    const bool cached = dev >= 0 && dev < 64;
    if (!cached || !done[dev].load(std::memory_order_acquire)) {
        XCT_CUDA_TRY(cudaFuncSetAttribute((const void *)adj_scatter_kernel<S, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)C::Smem));
        if (cached) done[dev].store(true, std::memory_order_release);
    }
    const int ntx = (g.nx + T - 1) / T, nty = (g.ny + T - 1) / T;
    adj_scatter_kernel<S, T><<<dim3(ntx * nty, 1, groups), C::Threads, C::Smem, st>>>(sino, img, trig, g, ntx, sub, step, nang,
                                                                                     base, scale);
    g_xct_launches.fetch_add(1, std::memory_order_relaxed);
    XCT_CUDA_TRY(cudaGetLastError());
    return XCT_OK;
}

// Modelled time of a launch over `groups` groups (SM cycles per angle): the CTAs one SM gets, times a
// CTA's cycles.  Scatter (T > 0): per group of eight rays (1.27 T / 8 of them, a half more for the ends)
// 120 instructions and, per step of four samples, 16 and 14 per slice (eff: idle lanes at the rays'
// ends), three instructions a cycle; measured 1930 cycles for S = 1, T = 64.  Gather: measured cycles per
// block (1024^2 x 720 angles).
double adj_cost(int nx, int ny, int S, int T, int groups, int sms)
{
    double cta;
    long long n;
    if (T > 0) {
        const double eff = T == 16 ? 1.6 : T == 32 ? 1.3 : T == 44 ? 1.21 : 1.155;
        cta = ((1.27 * T / 8 + 0.5) * (120 + 0.196 * T * eff * (16 + 14 * S)) + 0.02 * S * T * T) / 3;
        n = (long long)((nx + T - 1) / T) * ((ny + T - 1) / T);
    } else {
        const int BY = S <= 8 ? 16 : 20;
        cta = S == 4 ? 700 : S == 8 ? 840 : 1230;
        n = (long long)((nx + 30) / 31) * ((ny + BY - 2) / (BY - 1));
    }
    n *= groups;
    return (double)((n + sms - 1) / sms) * cta;
}

}  // namespace

int launch_adj_tiled(const KGeom &g, const float2 *trig, const float *sino, float *img, int dN, cudaStream_t st)
{
    return launch_adj_subset(g, trig, sino, img, dN, 0, 1, g.pa, nullptr, 0.0f, st);
}

int launch_adj_subset(const KGeom &g, const float2 *trig, const float *sino, float *img, int dN, int sub, int step,
                      int nang, const float *base, float scale, cudaStream_t st)
{
    // The form with the least modelled time per slice takes as many of its groups as the call has, then the
    // rest likewise: gather for groups of ten, eight and four (its candidate search is shared by the
    // group), scatter for one or two slices; large images prefer large tiles, small ones small tiles that
    // reach every SM.  With grouping off (by hand) every slice is scattered alone.
    struct Form {
        int S, T;  // T = 0: gather
        int (*run)(const KGeom &, const float2 *, const float *, float *, int, int, int, int, const float *, float,
                   cudaStream_t);
    };
    static const Form forms[] = {{10, 0, launch_adj_gather<10>},     {8, 0, launch_adj_gather<8>},
                                 {4, 0, launch_adj_gather<4>},       {2, 44, launch_adj_scatter<2, 44>},
                                 {2, 32, launch_adj_scatter<2, 32>}, {1, 64, launch_adj_scatter<1, 64>},
                                 {1, 44, launch_adj_scatter<1, 44>}, {1, 32, launch_adj_scatter<1, 32>},
                                 {1, 16, launch_adj_scatter<1, 16>}};
    const int sms = device_sm_count();
    while (dN > 0) {
        const Form *best = nullptr;
        double cost = 0.0;
        for (const Form &f : forms) {
            if (f.S > dN || (f.S > 1 && !g.fwd_group)) continue;
            const int groups = dN / f.S;
            const double c = adj_cost(g.nx, g.ny, f.S, f.T, groups, sms) / (groups * f.S);
            if (!best || c < cost) {
                best = &f;
                cost = c;
            }
        }
        const int groups = dN / best->S, n = groups * best->S;
        const int rc = best->run(g, trig, sino, img, groups, sub, step, nang, base, scale, st);
        if (rc) return rc;
        sino += (size_t)n * g.pa * g.px;
        img += (size_t)n * g.nx * g.ny;
        if (base) base += (size_t)n * g.nx * g.ny;
        dN -= n;
    }
    return XCT_OK;
}

XCT_CHECK_READER(xct_check_read_adj)
