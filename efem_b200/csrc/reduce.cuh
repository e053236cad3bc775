// Reductions of many values at once, in a fixed order (results repeat bitwise).
#pragma once
#include <cuda_runtime.h>

namespace efem {

// Sums of NV <= 32 values over a CTA of `Warps` warps: on return lane k < NV of
// warp 0 holds the total of value k.  A warp halves the number of values it
// carries with every exchange (about 2 NV shuffles in all instead of 5 NV), and
// the warps' sums meet in sh[Warps][32].
template <int NV, int Warps>
__device__ __forceinline__ double cta_sums(const double (&v)[NV], double (*sh)[32])
{
    constexpr int P = NV <= 1 ? 1 : NV <= 2 ? 2 : NV <= 4 ? 4 : NV <= 8 ? 8 : NV <= 16 ? 16 : 32;
    constexpr int L = P == 1 ? 0 : P == 2 ? 1 : P == 4 ? 2 : P == 8 ? 3 : P == 16 ? 4 : 5;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double a[P];
#pragma unroll
    for (int k = 0; k < P; k++) a[k] = k < NV ? v[k < NV ? k : 0] : 0.0;
#pragma unroll
    for (int s = 0; s < L; s++) {
        const int h = P >> (s + 1), o = 16 >> s;
        const bool up = lane & o;
#pragma unroll
        for (int k = 0; k < h; k++) {
            const double keep = up ? a[k + h] : a[k], send = up ? a[k] : a[k + h];
            a[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
#pragma unroll
    for (int o = 16 >> L; o > 0; o >>= 1) a[0] += __shfl_xor_sync(0xffffffffu, a[0], o);
    if ((lane & ((32 >> L) - 1)) == 0) sh[w][lane >> (5 - L)] = a[0];
    __syncthreads();
    double t = 0.0;
    if (w == 0 && lane < NV) {
#pragma unroll
        for (int q = 0; q < Warps; q++) t += sh[q][lane];
    }
    return t;
}

// The two-loop recursion's first loop (LBFGSMat.h:106-113) by one warp: lane k
// holds t = s_k . q0 of slot k, ys its s_k . y_k; slots are visited newest
// first from `loc`; G[k * ld + j] = s_k . y_j.  Returns alpha_k in lane k.
__device__ __forceinline__ double first_loop(double t, double ys, const double* G, int ld, int loc, int m, int ncorr)
{
    const int lane = threadIdx.x & 31;
    double alpha = 0.0;
    for (int i = 0; i < ncorr; i++) {
        const int j = loc - i < 0 ? loc - i + m : loc - i;
        const double al = __shfl_sync(0xffffffffu, t / ys, j);
        if (lane == j) alpha = al;
        if (lane < ncorr) t -= al * G[lane * ld + j];
    }
    return alpha;
}

// The second loop (LBFGSMat.h:121-128): lane k holds t = y_k . z0 and alpha_k;
// slots oldest first, ptr the slot after the newest.  Returns alpha - beta.
__device__ __forceinline__ double second_loop(double t, double ys, double alpha, const double* G, int ld, int ptr, int m, int ncorr)
{
    const int lane = threadIdx.x & 31;
    double coef = 0.0;
    for (int o = 0; o < ncorr; o++) {
        const int j = (((ptr - ncorr + o) % m) + m) % m;
        const double cf = __shfl_sync(0xffffffffu, alpha - t / ys, j);
        if (lane == j) coef = cf;
        if (lane < ncorr) t += cf * G[j * ld + lane];
    }
    return coef;
}

}  // namespace efem
