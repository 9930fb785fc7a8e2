// xct_ray.cuh -- the exact interval of a ray's samples inside a range of one coordinate.
#pragma once
#include <cuda_runtime.h>

__device__ __forceinline__ float ray_coord(int Y, float hd, float sl, float a)
{
    return fmaf((float)Y - hd, sl, a);
}

// First Y in [0, D] where the monotone predicate P holds (D if none), with the sentinels
// P(-1) = false, P(D) = true:  sl > 0: P(Y) = u(Y) >= b;  sl < 0: P(Y) = u(Y) < b,
// u(Y) = fma(Y - hd, sl, a).  The estimate from the real crossing point is checked with
// two exact evaluations; a binary search settles the rare cases it misses.
static __device__ __noinline__ int first_true_search(float b, float a, float sl, float hd, int D)
{
    const bool up = sl > 0.0f;
    int lo = 0, hi = D;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        const float u = ray_coord(mid, hd, sl, a);
        if (up ? (u >= b) : (u < b)) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

__device__ __forceinline__ int first_true(float b, float a, float sl, float inv_sl, float hd, int D)
{
    const bool up = sl > 0.0f;
    const float Df = (float)D;
    // the estimate as an integer-valued float in [0, D] (infinities clamp; NaN gives 0)
    const float Yf = fminf(fmaxf(ceilf(fmaf(b - a, inv_sl, hd)), 0.0f), Df);
    const float Yc = Yf - hd;  // exact, as the samples' own
    const float ul = fmaf(Yc - 1.0f, sl, a), uh = fmaf(Yc, sl, a);
    const bool pl = Yf > 0.0f && (ul >= b) == up;
    const bool ph = Yf >= Df || (uh >= b) == up;
    if (!pl && ph) return (int)Yf;
    return first_true_search(b, a, sl, hd, D);
}
