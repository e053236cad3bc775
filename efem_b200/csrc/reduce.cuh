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

// max that keeps a NaN (fmax drops it): a non-finite residual or solution
// must show in its infinity norm (Integrator.cpp:28-34 tests for it)
__device__ __forceinline__ double nan_max(double a, double b) { return (b > a || b != b) ? b : a; }

// The same for NS sums followed by NM maxima of values >= 0: lane k < NS + NM
template <int NS, int NM, int Warps>
__device__ __forceinline__ double cta_totals(const double (&v)[NS + NM], double (*sh)[32])
{
    static_assert(NM == 0 || (NS <= 16 && NM <= 16), "columns of sh");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double a[NS];
#pragma unroll
    for (int k = 0; k < NS; k++) a[k] = v[k];
#pragma unroll
    for (int k = 0; k < NM; k++) {
        double b = v[NS + k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) b = nan_max(b, __shfl_xor_sync(0xffffffffu, b, o));
        if (lane == 0) sh[w][16 + k] = b;
    }
    double t = cta_sums<NS, Warps>(a, sh);
    if (NM > 0 && w == 0 && lane >= NS && lane < NS + NM) {
#pragma unroll
        for (int q = 0; q < Warps; q++) t = nan_max(t, sh[q][16 + lane - NS]);
    }
    return t;
}

// The two-loop recursion's first loop (LBFGSMat.h:106-113) by one warp: lane k
// holds u = (s_k . q0) / ys_k of slot k and G[k * ld + j] = (s_k . y_j) / ys_k;
// slots are visited newest first from `loc`.  Returns alpha_k in lane k.  The
// divisions by ys_k = s_k . y_k are done beforehand, all at once: one in every
// step of the chain made a recursion of six pairs 4.3 us.
__device__ __forceinline__ double first_loop(double u, const double* G, int ld, int loc, int m, int ncorr)
{
    const int lane = threadIdx.x & 31;
    double alpha = 0.0;
    for (int i = 0, j = loc; i < ncorr; i++, j = j == 0 ? m - 1 : j - 1) {
        const double g = lane < ncorr ? G[lane * ld + j] : 0.0;
        const double al = __shfl_sync(0xffffffffu, u, j);
        if (lane == j) alpha = al;
        u -= al * g;
    }
    return alpha;
}

// The second loop (LBFGSMat.h:121-128): lane k holds w = (y_k . z0) / ys_k and
// alpha_k, G[j * ld + k] = (s_j . y_k) / ys_k; slots oldest first, ptr the slot
// after the newest.  Returns alpha - beta.
__device__ __forceinline__ double second_loop(double w, double alpha, const double* G, int ld, int ptr, int m, int ncorr)
{
    const int lane = threadIdx.x & 31;
    double coef = 0.0;
    for (int o = 0, j = (((ptr - ncorr) % m) + m) % m; o < ncorr; o++, j = j == m - 1 ? 0 : j + 1) {
        const double g = lane < ncorr ? G[j * ld + lane] : 0.0;
        const double cf = __shfl_sync(0xffffffffu, alpha - w, j);
        if (lane == j) coef = cf;
        w += cf * g;
    }
    return coef;
}

}  // namespace efem
