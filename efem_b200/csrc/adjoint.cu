// True tangent, adjoint solve and parameter sensitivities.  The reference has
// none of these (it only ever forms the approximate Jacobian, see
// src/fe/ElementConstraint.cpp:164-205); they are built on its residual
// (ElementConstraint.cpp:139-162, ExternalConstraint.cpp:829-959):
//
//   K(u) v      the directional derivative of R at u along v, the residual's
//               phases with the laws differentiated by hand (piola_tangent);
//   K(u)^T w    the element part of K is the Hessian of the stored energy and
//               is symmetric, so K_el^T w = K_el w; the pressure part is not
//               (follower and directed loads are not conservative) and is
//               transposed face by face, point by point;
//   dR/dtheta   the residual on forward-mode dual numbers (value + derivative),
//               with the seed on a material constant
//               (C10, C01, C20, C30, D1 of one material) or on the scale of one
//               pressure load;
//   adjoint     K(u)^T lambda = dJ/du by restarted GMRES, right-preconditioned
//               with the approximate-Jacobian Cholesky factor H0 of the
//               solve; then dJ/dtheta_k = -lambda . dR/dtheta_k.
//
// Parameter order: for every material slot of the model (its material
// table), C10, C01, C20, C30, D1; then one scale per pressure load in input
// order (a follower load's pressure value, a directed load's vector scale).
#include <cuda_runtime.h>


#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "dual.cuh"
#include "efem_internal.h"
#include "mechanics.cuh"

namespace efem {

template <>
__device__ __forceinline__ Dual drcbrt<Dual>(Dual x)
{
    const double r = rcbrt(x.v);
    return Dual(r, -(1.0 / 3.0) * (r * r) * (r * r) * x.d);  // d J^{-1/3} / dJ = -J^{-4/3} / 3
}

namespace {

constexpr int kBlock = 128;
constexpr int kVec = 256;        // threads of the vector kernels
constexpr int kDotBlocks = 128;  // CTAs per dot product
constexpr int kRestart = 100;    // GMRES restart length

struct TanElemArgs {
    int n, n_free;
    const int* __restrict__ conn;   // [NEN][n]
    const int* __restrict__ mat;    // [n]
    const double* __restrict__ vol;
    const double* __restrict__ J0inv;
    const double* __restrict__ dN;
    const double* __restrict__ gw;
    const MatParams<Dual>* __restrict__ mats;  // k_elem_tangent: one constant seeded
    const double* __restrict__ u;
    const double* __restrict__ v;   // direction (k_tangent)
    double* __restrict__ out;       // += derivative of r
};

// elements per CTA of the tangent kernels (two values per unknown in shared memory)
__host__ __device__ constexpr int tan_epb(int ngp) { return (kBlock / ngp) < 1 ? 1 : ((kBlock / ngp) > 32 ? 32 : kBlock / ngp); }

// The element residual of residual.cu on dual numbers, the seed on a material
// constant: out += d r_el / d theta.
template <int NEN, int NGP>
__global__ void __launch_bounds__(kBlock) k_elem_tangent(TanElemArgs a)
{
    constexpr int EPB = tan_epb(NGP);
    __shared__ Dual s_u[EPB][NEN][3];
    __shared__ Dual s_S[EPB][NGP][9];
    __shared__ double s_dN[NGP][NEN][3];
    __shared__ int s_node[EPB][NEN];
    const int tid = threadIdx.x;
    for (int i = tid; i < NGP * NEN * 3; i += kBlock) (&s_dN[0][0][0])[i] = a.dN[i];
    const int e0 = blockIdx.x * EPB;
    for (int i = tid; i < EPB * NEN; i += kBlock) {
        const int el = i % EPB, nd = i / EPB, e = e0 + el;
        int node = a.n_free;
        Dual x[3];
        if (e < a.n) {
            node = a.conn[static_cast<size_t>(nd) * a.n + e];
            if (node < a.n_free)
#pragma unroll
                for (int c = 0; c < 3; c++) x[c] = Dual(a.u[3 * node + c]);
        }
        s_node[el][nd] = node;
#pragma unroll
        for (int c = 0; c < 3; c++) s_u[el][nd][c] = x[c];
    }
    __syncthreads();
    if (tid < EPB * NGP) {
        const int el = tid / NGP, g = tid % NGP, e = e0 + el;
        if (e < a.n) {
            Dual A[9];
            for (int q = 0; q < NEN; q++)
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int k = 0; k < 3; k++) A[3 * i + k] += s_u[el][q][i] * Dual(s_dN[g][q][k]);
            const double* Ji = a.J0inv + (static_cast<size_t>(e) * NGP + g) * 9;
            Dual H[9];
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int j = 0; j < 3; j++)
                    H[3 * i + j] = A[3 * i] * Dual(Ji[j]) + A[3 * i + 1] * Dual(Ji[3 + j]) + A[3 * i + 2] * Dual(Ji[6 + j]);
            const MatParams<Dual> mp = a.mats[a.mat[e]];
            Dual P[9];
            piola(mp, H, P);
            const Dual wv = Dual(a.vol[e] * a.gw[g]);
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int j = 0; j < 3; j++)
                    s_S[el][g][3 * i + j] =
                        wv * (P[3 * i] * Dual(Ji[3 * j]) + P[3 * i + 1] * Dual(Ji[3 * j + 1]) + P[3 * i + 2] * Dual(Ji[3 * j + 2]));
        }
    }
    __syncthreads();
    for (int i = tid; i < EPB * NEN; i += kBlock) {
        const int el = i % EPB, nd = i / EPB, e = e0 + el;
        if (e >= a.n) continue;
        const int node = s_node[el][nd];
        if (node >= a.n_free) continue;
        double r[3] = { 0, 0, 0 };
        for (int g = 0; g < NGP; g++) {
            const double* d = s_dN[g][nd];
            const Dual* S = s_S[el][g];
#pragma unroll
            for (int c = 0; c < 3; c++) r[c] += S[3 * c].d * d[0] + S[3 * c + 1].d * d[1] + S[3 * c + 2].d * d[2];
        }
#pragma unroll
        for (int c = 0; c < 3; c++) atomicAdd(a.out + 3 * node + c, r[c]);
    }
}

struct TanFaceArgs {
    int n, n_free;
    int gmax;                           // most points of a face in the set
    const int* __restrict__ conn;
    const int* __restrict__ table;
    const int* __restrict__ load_idx;
    const double* __restrict__ A0;
    const double* __restrict__ J0inv;
    const double* __restrict__ load;
    const int* __restrict__ t_ngp;
    const double* __restrict__ t_w;
    const double* __restrict__ t_N;
    const double* __restrict__ t_dN;
    const double* __restrict__ u;
    const double* __restrict__ v;       // tangent: direction, or the vector K^T is applied to
    const double* __restrict__ dscale;  // k_face_tangent: per pressure load, the derivative of its scale
    double* __restrict__ out;
};

constexpr int face_epb(int nen) { return nen >= 20 ? 8 : nen >= 8 ? 16 : 32; }

template <int NEN>
struct TanFaceSmem {
    static constexpr int EPB = face_epb(NEN);
    double u[EPB][(NEN * 3) | 1], v[EPB][(NEN * 3) | 1];
    double q[EPB][(MAX_FGP * 9) | 1];  // per face point: d(cof F A0) or its norm (forward); ds/d(sum_q u_q dN_q) (transpose)
    int node[EPB][NEN];
    int table[EPB], ngp[EPB];
};

// out -= K_face v (transpose: K_face^T v) for one tile of faces, in the phases
// of the face residual.  With H = du/dX at a face point and cof F = I + B(H),
//   forward    d(cof F A0) = dB A0, dB the derivative of B along dH = dv/dX;
//   transpose  s = lambda . (cof F A0) with lambda = sum_q w N_q (p v_q) (for a
//              directed load lambda = (sum_q w N_q L . v_q) cof F A0 / |cof F A0|):
//              ds/dH_ij = delta_ij (lambda . A0) - A0_i lambda_j + ([lambda]x H [A0]x^T)_ij
//              (cof is bilinear: its derivative along E_ij contracts two permutation
//              symbols), then back through H to the nodes.
// In place of one pass of dual numbers over the face per unknown (3 NEN of
// them), or of stored 3 NEN x 3 NEN blocks read in every product.
template <int NEN>
__device__ void tan_face_tile(const TanFaceArgs& a, int tile, TanFaceSmem<NEN>& sm, bool transpose)
{
    constexpr int EPB = face_epb(NEN);
    const int tid = threadIdx.x, fb = tile * EPB;
    if (tid < EPB) {
        const int t = fb + tid < a.n ? a.table[fb + tid] : 0;
        sm.table[tid] = t;
        sm.ngp[tid] = a.t_ngp[t];
    }
    for (int i = tid; i < EPB * NEN; i += kBlock) {
        const int el = i % EPB, q = i / EPB, f = fb + el;
        int node = a.n_free;
        double x[3] = { 0, 0, 0 }, y[3] = { 0, 0, 0 };
        if (f < a.n) {
            node = a.conn[static_cast<size_t>(q) * a.n + f];
            if (node < a.n_free)
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    x[c] = a.u[3 * node + c];
                    y[c] = a.v[3 * node + c];
                }
        }
        sm.node[el][q] = node;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            sm.u[el][3 * q + c] = x[c];
            sm.v[el][3 * q + c] = y[c];
        }
    }
    __syncthreads();
    for (int i = tid; i < EPB * a.gmax; i += kBlock) {
        const int el = i / a.gmax, g = i - el * a.gmax, f = fb + el;
        if (f >= a.n) break;
        if (g >= sm.ngp[el]) continue;
        const size_t tg = static_cast<size_t>(sm.table[el]) * MAX_FGP + g;
        const double* dN = a.t_dN + tg * NEN * 3;
        const double* L = a.load + 4 * f;
        const bool directed = L[0] != 0.0;
        double Ji[9], A0[3];
#pragma unroll
        for (int k = 0; k < 9; k++) Ji[k] = a.J0inv[(static_cast<size_t>(f) * MAX_FGP + g) * 9 + k];
#pragma unroll
        for (int k = 0; k < 3; k++) A0[k] = a.A0[3 * f + k];
        double A[9] = {}, D[9] = {}, lam[3] = {};
#pragma unroll 2
        for (int q = 0; q < NEN; q++) {
            const double wn = a.t_w[sm.table[el] * MAX_FGP + g] * a.t_N[tg * NEN + q];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                lam[c] += wn * sm.v[el][3 * q + c];
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    A[3 * c + k] += sm.u[el][3 * q + c] * dN[3 * q + k];
                    if (!transpose) D[3 * c + k] += sm.v[el][3 * q + c] * dN[3 * q + k];
                }
            }
        }
        double H[9];
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
            for (int j = 0; j < 3; j++) H[3 * c + j] = A[3 * c] * Ji[j] + A[3 * c + 1] * Ji[3 + j] + A[3 * c + 2] * Ji[6 + j];
        Kin<double> k;
        kinematics(H, k);
        double cA[3];
#pragma unroll
        for (int c = 0; c < 3; c++) cA[c] = A0[c] + k.B[3 * c] * A0[0] + k.B[3 * c + 1] * A0[1] + k.B[3 * c + 2] * A0[2];
        const double nrm = ::sqrt(cA[0] * cA[0] + cA[1] * cA[1] + cA[2] * cA[2]), inrm = nrm > 0.0 ? 1.0 / nrm : 0.0;
        double* out = sm.q[el] + 9 * g;
        if (transpose) {
            if (directed) {
                const double mu = (L[1] * lam[0] + L[2] * lam[1] + L[3] * lam[2]) * inrm;
#pragma unroll
                for (int c = 0; c < 3; c++) lam[c] = mu * cA[c];
            } else {
#pragma unroll
                for (int c = 0; c < 3; c++) lam[c] *= L[1];
            }
            // T = [lam]x H (rows), G = T [A0]x^T + (lam . A0) I - A0 lam^T
            double T[9], G[9];
#pragma unroll
            for (int j = 0; j < 3; j++) {
                T[j] = lam[2] * H[3 + j] - lam[1] * H[6 + j];
                T[3 + j] = lam[0] * H[6 + j] - lam[2] * H[j];
                T[6 + j] = lam[1] * H[j] - lam[0] * H[3 + j];
            }
            const double la = lam[0] * A0[0] + lam[1] * A0[1] + lam[2] * A0[2];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                G[3 * c] = A0[2] * T[3 * c + 1] - A0[1] * T[3 * c + 2];
                G[3 * c + 1] = A0[0] * T[3 * c + 2] - A0[2] * T[3 * c];
                G[3 * c + 2] = A0[1] * T[3 * c] - A0[0] * T[3 * c + 1];
#pragma unroll
                for (int j = 0; j < 3; j++) G[3 * c + j] += (c == j ? la : 0.0) - A0[c] * lam[j];
            }
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int m = 0; m < 3; m++)
                    out[3 * c + m] = G[3 * c] * Ji[3 * m] + G[3 * c + 1] * Ji[3 * m + 1] + G[3 * c + 2] * Ji[3 * m + 2];
        } else {
            double d[9];
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int j = 0; j < 3; j++) d[3 * c + j] = D[3 * c] * Ji[j] + D[3 * c + 1] * Ji[3 + j] + D[3 * c + 2] * Ji[6 + j];
            double dA[3];
            const double t = d[0] + d[4] + d[8];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const int p = 3 * ((c + 1) % 3), q = 3 * ((c + 2) % 3);
                dA[c] = t * A0[c];
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    const int x = (j + 1) % 3, y = (j + 2) % 3;
                    dA[c] += (d[p + x] * H[q + y] + H[p + x] * d[q + y] - d[p + y] * H[q + x] - H[p + y] * d[q + x] - d[3 * j + c]) * A0[j];
                }
            }
            if (directed) dA[0] = (cA[0] * dA[0] + cA[1] * dA[1] + cA[2] * dA[2]) * inrm;
#pragma unroll
            for (int c = 0; c < 3; c++) out[c] = dA[c];
        }
    }
    __syncthreads();
    for (int i = tid; i < EPB * NEN; i += kBlock) {
        const int el = i % EPB, q = i / EPB, f = fb + el;
        if (f >= a.n) continue;
        const int node = sm.node[el][q];
        if (node >= a.n_free) continue;
        const int t = sm.table[el], ngp = sm.ngp[el];
        const double* L = a.load + 4 * f;
        double s[3] = { 0, 0, 0 };
        for (int g = 0; g < ngp; g++) {
            const size_t tg = static_cast<size_t>(t) * MAX_FGP + g;
            const double* Q = sm.q[el] + 9 * g;
            if (transpose) {
                const double* dN = a.t_dN + (tg * NEN + q) * 3;
                const double d0 = dN[0], d1 = dN[1], d2 = dN[2];
#pragma unroll
                for (int c = 0; c < 3; c++) s[c] += Q[3 * c] * d0 + Q[3 * c + 1] * d1 + Q[3 * c + 2] * d2;
            } else {
                const double wn = a.t_w[t * MAX_FGP + g] * a.t_N[tg * NEN + q];
#pragma unroll
                for (int c = 0; c < 3; c++) s[c] += wn * Q[c];
            }
        }
        if (!transpose) {
            const bool directed = L[0] != 0.0;
            const double s0 = s[0];
#pragma unroll
            for (int c = 0; c < 3; c++) s[c] = directed ? L[1 + c] * s0 : L[1] * s[c];
        }
#pragma unroll
        for (int c = 0; c < 3; c++) atomicAdd(a.out + 3 * node + c, -s[c]);
    }
}

template <int NEN, int NGP>
struct TanElemSmem {
    static constexpr int EPB = tan_epb(NGP);
    double u[EPB][(NEN * 3) | 1], v[EPB][(NEN * 3) | 1];  // rows of odd length: no bank conflicts over elements
    double S[EPB][(NGP * 9) | 1];
    double dN[NGP][(NEN * 3) | 1];
    int node[EPB][NEN | 1];
};

// out += K_el v, the derivative of the element residual of residual.cu along
// v, in its three phases with dP = dP/dH : dH by hand (piola_tangent) in place
// of dual numbers; the first n_face_tiles CTAs take the faces.  Bound by
// latency: 16 warps per SM with the neo-Hookean and Yeoh laws (124 to 126
// registers; issue slots 29% busy, a third of the stalls on loads), 12 with
// Mooney-Rivlin and in blocks of mixed laws (164 to 168).  C3D10 Yeoh finger,
// transpose product with the chamber faces: 32 us (cold), where the elements on
// dual numbers took 77 us (240 registers, 8 warps per SM) and the faces 68 us
// more; the products of an adjoint solve, which read stored Gauss-point
// tangents (131 MB) and face blocks, are no slower without them.
template <int NEN, int NGP, int MT>
__global__ void __launch_bounds__(kBlock) k_tangent(TanElemArgs a, const MatParams<double>* __restrict__ mats,
    TanFaceArgs fa, int n_face_tiles, int transpose)
{
    constexpr int EPB = tan_epb(NGP);
    __shared__ union Smem {
        TanElemSmem<NEN, NGP> e;
        TanFaceSmem<NEN> f;
        __device__ Smem() {}
    } smem;
    if (static_cast<int>(blockIdx.x) < n_face_tiles) {
        tan_face_tile<NEN>(fa, blockIdx.x, smem.f, transpose != 0);
        return;
    }
    auto& sm = smem.e;
    const int tid = threadIdx.x, e0 = (static_cast<int>(blockIdx.x) - n_face_tiles) * EPB;
    for (int i = tid; i < NGP * NEN * 3; i += kBlock) sm.dN[i / (NEN * 3)][i % (NEN * 3)] = a.dN[i];
    for (int i = tid; i < EPB * NEN; i += kBlock) {
        const int el = i % EPB, nd = i / EPB, e = e0 + el;
        int node = a.n_free;
        double x[3] = { 0, 0, 0 }, y[3] = { 0, 0, 0 };
        if (e < a.n) {
            node = a.conn[static_cast<size_t>(nd) * a.n + e];
            if (node < a.n_free)
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    x[c] = a.u[3 * node + c];
                    y[c] = a.v[3 * node + c];
                }
        }
        sm.node[el][nd] = node;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            sm.u[el][3 * nd + c] = x[c];
            sm.v[el][3 * nd + c] = y[c];
        }
    }
    __syncthreads();
    if (tid < EPB * NGP) {
        const int el = tid / NGP, g = tid % NGP, e = e0 + el;
        if (e < a.n) {
            const double* Jp = a.J0inv + (static_cast<size_t>(e) * NGP + g) * 9;
            double H[9], dH[9];
            {
                double Ji[9], A[9] = {}, D[9] = {};
#pragma unroll
                for (int k = 0; k < 9; k++) Ji[k] = __ldg(Jp + k);
#pragma unroll 2
                for (int q = 0; q < NEN; q++)
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        const double d = sm.dN[g][3 * q + k];
#pragma unroll
                        for (int i = 0; i < 3; i++) {
                            A[3 * i + k] += sm.u[el][3 * q + i] * d;
                            D[3 * i + k] += sm.v[el][3 * q + i] * d;
                        }
                    }
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int j = 0; j < 3; j++) {
                        H[3 * i + j] = A[3 * i] * Ji[j] + A[3 * i + 1] * Ji[3 + j] + A[3 * i + 2] * Ji[6 + j];
                        dH[3 * i + j] = D[3 * i] * Ji[j] + D[3 * i + 1] * Ji[3 + j] + D[3 * i + 2] * Ji[6 + j];
                    }
            }
            double dP[9];
            piola_tangent<MT>(mats[__ldg(a.mat + e)], H, dH, dP);
            const double wv = __ldg(a.vol + e) * __ldg(a.gw + g);
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const double j0 = __ldg(Jp + 3 * j), j1 = __ldg(Jp + 3 * j + 1), j2 = __ldg(Jp + 3 * j + 2);
#pragma unroll
                for (int i = 0; i < 3; i++)
                    sm.S[el][9 * g + 3 * i + j] = wv * (dP[3 * i] * j0 + dP[3 * i + 1] * j1 + dP[3 * i + 2] * j2);
            }
        }
    }
    __syncthreads();
    for (int i = tid; i < EPB * NEN; i += kBlock) {
        const int el = i % EPB, nd = i / EPB, e = e0 + el;
        if (e >= a.n) continue;
        const int node = sm.node[el][nd];
        if (node >= a.n_free) continue;
        double r[3] = { 0, 0, 0 };
#pragma unroll 2
        for (int g = 0; g < NGP; g++) {
            const double d0 = sm.dN[g][3 * nd], d1 = sm.dN[g][3 * nd + 1], d2 = sm.dN[g][3 * nd + 2];
            const double* S = sm.S[el] + 9 * g;
#pragma unroll
            for (int c = 0; c < 3; c++) r[c] += S[3 * c] * d0 + S[3 * c + 1] * d1 + S[3 * c + 2] * d2;
        }
#pragma unroll
        for (int c = 0; c < 3; c++) atomicAdd(a.out + 3 * node + c, r[c]);
    }
}

// faces without an element block of their kind to go with
template <int NEN>
__global__ void __launch_bounds__(kBlock) k_tangent_faces(TanFaceArgs a, int transpose)
{
    __shared__ TanFaceSmem<NEN> sm;
    tan_face_tile<NEN>(a, blockIdx.x, sm, transpose != 0);
}

// Nodal forces f_q (all NEN nodes, dual) of face f with node displacements uu,
// as in the face residual of residual.cu; the load value's derivative is
// dscale times the load (pressure value, or directed vector).
template <int NEN>
__device__ void face_forces(const TanFaceArgs& a, int f, const Dual (*uu)[3], Dual (*fq)[3])
{
    const int t = a.table[f];
    const int ngp = a.t_ngp[t];
    const double* L = a.load + 4 * f;
    const bool directed = L[0] != 0.0;
    const double ds = a.dscale[a.load_idx[f]];
    Dual cA[MAX_FGP][3];
    for (int g = 0; g < ngp; g++) {
        const double* dN = a.t_dN + (static_cast<size_t>(t) * MAX_FGP + g) * NEN * 3;
        Dual A[9];
        for (int q = 0; q < NEN; q++)
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int k = 0; k < 3; k++) A[3 * i + k] += uu[q][i] * Dual(dN[3 * q + k]);
        const double* Ji = a.J0inv + (static_cast<size_t>(f) * MAX_FGP + g) * 9;
        Dual H[9];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++)
                H[3 * i + j] = A[3 * i] * Dual(Ji[j]) + A[3 * i + 1] * Dual(Ji[3 + j]) + A[3 * i + 2] * Dual(Ji[6 + j]);
        Kin<Dual> k;
        kinematics(H, k);
        const Dual A0[3] = { Dual(a.A0[3 * f]), Dual(a.A0[3 * f + 1]), Dual(a.A0[3 * f + 2]) };
#pragma unroll
        for (int i = 0; i < 3; i++) cA[g][i] = A0[i] + k.B[3 * i] * A0[0] + k.B[3 * i + 1] * A0[1] + k.B[3 * i + 2] * A0[2];
        if (directed) cA[g][0] = sqrt(cA[g][0] * cA[g][0] + cA[g][1] * cA[g][1] + cA[g][2] * cA[g][2]);
    }
    for (int q = 0; q < NEN; q++) {
        Dual s[3];
        for (int g = 0; g < ngp; g++) {
            const Dual wn = Dual(a.t_w[t * MAX_FGP + g] * a.t_N[(static_cast<size_t>(t) * MAX_FGP + g) * NEN + q]);
            if (directed) {
                s[0] += wn * cA[g][0];
            } else {
#pragma unroll
                for (int i = 0; i < 3; i++) s[i] += wn * cA[g][i];
            }
        }
        if (directed) {
#pragma unroll
            for (int i = 0; i < 3; i++) fq[q][i] = Dual(L[1 + i]) * s[0] + Dual(0.0, ds * L[1 + i] * s[0].v);
        } else {
#pragma unroll
            for (int i = 0; i < 3; i++) fq[q][i] = Dual(L[1]) * s[i] + Dual(0.0, ds * s[i].v);
        }
    }
}

// out -= d f / d scale (the face part of R is -f)
template <int NEN>
__global__ void __launch_bounds__(kBlock) k_face_tangent(TanFaceArgs a)
{
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= a.n) return;
    int node[NEN];
    Dual uu[NEN][3];
    for (int q = 0; q < NEN; q++) {
        node[q] = a.conn[static_cast<size_t>(q) * a.n + f];
        const bool fr = node[q] < a.n_free;
#pragma unroll
        for (int c = 0; c < 3; c++) uu[q][c] = Dual(fr ? a.u[3 * node[q] + c] : 0.0);
    }
    Dual fq[NEN][3];
    face_forces<NEN>(a, f, uu, fq);
    for (int q = 0; q < NEN; q++) {
        if (node[q] >= a.n_free) continue;
#pragma unroll
        for (int c = 0; c < 3; c++) atomicAdd(a.out + 3 * node[q] + c, -fq[q][c].d);
    }
}

// ---------------------------------------------------------------- vectors
// per-CTA partial sums of the dot products x_k . y (k < nk) into
// part[k][blockIdx.x]; a CTA takes kDotRows rows, so y is read once for them
constexpr int kDotRows = 4;
__global__ void __launch_bounds__(kVec) k_dots(const double* __restrict__ X, size_t ldx, int nk,
    const double* __restrict__ y, size_t n, double* __restrict__ part)
{
    __shared__ double sh[kDotRows][kVec / 32];
    const int k0 = blockIdx.y * kDotRows, rows = min(kDotRows, nk - k0);
    const double* x = X + k0 * ldx;
    double s[kDotRows] = {};
#pragma unroll 2
    for (size_t i = blockIdx.x * (size_t)kVec + threadIdx.x; i < n; i += (size_t)gridDim.x * kVec) {
        const double yi = y[i];
#pragma unroll
        for (int k = 0; k < kDotRows; k++)
            if (k < rows) s[k] += x[k * ldx + i] * yi;
    }
#pragma unroll
    for (int k = 0; k < kDotRows; k++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
        if ((threadIdx.x & 31) == 0) sh[k][threadIdx.x >> 5] = s[k];
    }
    __syncthreads();
    if (threadIdx.x < rows) {
        double t = 0.0;
        for (int q = 0; q < kVec / 32; q++) t += sh[threadIdx.x][q];
        part[static_cast<size_t>(k0 + threadIdx.x) * gridDim.x + blockIdx.x] = t;
    }
}

// y += sum_k c_k x_k, two entries per thread (16-byte loads; ldx and n even,
// y and X 16-byte aligned)
__global__ void __launch_bounds__(kVec) k_axpys2(double* __restrict__ y, const double* __restrict__ X, size_t ldx, int nk,
    const double* __restrict__ c, size_t n)
{
    const size_t n2 = n / 2, ld2 = ldx / 2;
    const double2* X2 = reinterpret_cast<const double2*>(X);
    double2* y2 = reinterpret_cast<double2*>(y);
    for (size_t i = blockIdx.x * (size_t)kVec + threadIdx.x; i < n2; i += (size_t)gridDim.x * kVec) {
        double2 s0 = y2[i], s1 = make_double2(0.0, 0.0), s2 = s1, s3 = s1;
        int k = 0;
        for (; k + 4 <= nk; k += 4) {
            const double2 a = X2[k * ld2 + i], b = X2[(k + 1) * ld2 + i];
            const double2 d = X2[(k + 2) * ld2 + i], e = X2[(k + 3) * ld2 + i];
            s0.x += c[k] * a.x;
            s0.y += c[k] * a.y;
            s1.x += c[k + 1] * b.x;
            s1.y += c[k + 1] * b.y;
            s2.x += c[k + 2] * d.x;
            s2.y += c[k + 2] * d.y;
            s3.x += c[k + 3] * e.x;
            s3.y += c[k + 3] * e.y;
        }
        for (; k < nk; k++) {
            const double2 a = X2[k * ld2 + i];
            s0.x += c[k] * a.x;
            s0.y += c[k] * a.y;
        }
        y2[i] = make_double2((s0.x + s1.x) + (s2.x + s3.x), (s0.y + s1.y) + (s2.y + s3.y));
    }
}

// y += sum_k c_k x_k (coefficients in device memory)
__global__ void __launch_bounds__(kVec) k_axpys(double* __restrict__ y, const double* __restrict__ X, size_t ldx, int nk,
    const double* __restrict__ c, size_t n)
{
    for (size_t i = blockIdx.x * (size_t)kVec + threadIdx.x; i < n; i += (size_t)gridDim.x * kVec) {
        // four independent sums keep four loads of X in flight per thread
        double s0 = y[i], s1 = 0.0, s2 = 0.0, s3 = 0.0;
        int k = 0;
        for (; k + 4 <= nk; k += 4) {
            s0 += c[k] * X[k * ldx + i];
            s1 += c[k + 1] * X[(k + 1) * ldx + i];
            s2 += c[k + 2] * X[(k + 2) * ldx + i];
            s3 += c[k + 3] * X[(k + 3) * ldx + i];
        }
        for (; k < nk; k++) s0 += c[k] * X[k * ldx + i];
        y[i] = (s0 + s1) + (s2 + s3);
    }
}

// one warp per row k < nk: s_k = sum of part[k][0..nb) in order; hacc[k] = s_k
// (accumulate: hacc[k] += s_k) and coef[k] = -s_k
__global__ void k_rows_reduce(const double* __restrict__ part, int nk, int nb, double* __restrict__ hacc,
    double* __restrict__ coef, int accumulate)
{
    const int k = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (k >= nk) return;
    double s = 0.0;
    for (int b = lane; b < nb; b += 32) s += part[static_cast<size_t>(k) * nb + b];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
        hacc[k] = accumulate ? hacc[k] + s : s;
        coef[k] = -s;
    }
}

// The middle of two Gram-Schmidt passes in one sweep over the basis:
//   w += sum_k coef_k v_k  (the first pass's update, coef = -h)   and
//   part[k] = v_k . w      (the second pass's products, with the updated w),
// or, with Norm, the second pass's update and part = w . w beside it.
// A CTA takes 64 entries of every vector at a time; warp q holds the rows
// k = q mod 8 and a lane two entries, so a thread uses the values that it
// loaded itself for both, from registers, and only the eight partial updates
// of an entry meet in shared memory.  With 64 vectors of 240 600 entries
// (123 MB) 27 us, 4.5 TB/s: bound by the loads in flight (16 warps an SM of 122
// registers, 45% of the stalls on loads) below HBM's rate.  As two updates and two products by
// themselves (36 + 20 us each; the basis read four times) an iteration's
// orthogonalisation took 140 us at the average 64 vectors, now 85.
constexpr int kGsTile = 64;
constexpr int kGsRows = 104;         // most basis vectors (kRestart + 1, rounded up to the warps)
constexpr int kGsPer = kGsRows / 8;  // rows per warp
constexpr int kGsBlocks = 2 * kSMs, kGsNormBlocks = 3 * kSMs;

template <bool Norm>
__global__ void __launch_bounds__(kVec, Norm ? 3 : 2) k_gs_update(double* __restrict__ w, const double* __restrict__ V, size_t ldv,
    int nk, const double* __restrict__ coef, size_t n, double* __restrict__ part)
{
    __shared__ double sw[2][8][kGsTile], sc[kGsRows];
    const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;
    for (int k = threadIdx.x; k < kGsRows; k += kVec) sc[k] = k < nk ? coef[k] : 0.0;
    __syncthreads();
    const size_t nt = (n + kGsTile - 1) / kGsTile;
    double acc[Norm ? 1 : kGsPer] = {};
    int b = 0;
    for (size_t t = blockIdx.x; t < nt; t += gridDim.x, b ^= 1) {
        const size_t i = t * kGsTile + lane;
        const bool on0 = i < n, on1 = i + 32 < n;
        const double* v = V + static_cast<size_t>(q) * ldv + i;
        double x0[kGsPer], x1[kGsPer];
#pragma unroll
        for (int e = 0; e < kGsPer; e++) {
            const bool k = q + 8 * e < nk;
            x0[e] = k && on0 ? v[8 * e * ldv] : 0.0;
            x1[e] = k && on1 ? v[8 * e * ldv + 32] : 0.0;
        }
        double s0 = q == 0 && on0 ? w[i] : 0.0, s1 = q == 0 && on1 ? w[i + 32] : 0.0;
#pragma unroll
        for (int e = 0; e < kGsPer; e++) {
            const double c = sc[q + 8 * e];
            s0 += c * x0[e];
            s1 += c * x1[e];
        }
        sw[b][q][lane] = s0;
        sw[b][q][lane + 32] = s1;
        __syncthreads();
        double u0 = 0.0, u1 = 0.0;
#pragma unroll
        for (int h = 0; h < 8; h++) {
            u0 += sw[b][h][lane];
            u1 += sw[b][h][lane + 32];
        }
        if (q == 0 && on0) w[i] = u0;
        if (q == 0 && on1) w[i + 32] = u1;
        if constexpr (Norm) {
            acc[0] += u0 * u0 + u1 * u1;  // the same in every warp
        } else {
#pragma unroll
            for (int e = 0; e < kGsPer; e++) acc[e] += x0[e] * u0 + x1[e] * u1;
        }
    }
    if constexpr (Norm) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
        if (threadIdx.x == 0) part[blockIdx.x] = acc[0];
    } else {
#pragma unroll
        for (int e = 0; e < kGsPer; e++) {
            double s = acc[e];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0 && q + 8 * e < nk) part[static_cast<size_t>(q + 8 * e) * gridDim.x + blockIdx.x] = s;
        }
    }
}

// *s = sqrt(sum of part[0..nb)) and y = x / *s (0 when that is 0), twice: the
// new basis vector and the copy of it that H0 is applied to in place.  Every
// CTA adds the partial sums for itself, in the same order.
__global__ void __launch_bounds__(kVec) k_gs_scale(double* __restrict__ y, double* __restrict__ z,
    const double* __restrict__ x, const double* __restrict__ part, int nb, double* __restrict__ s, size_t n)
{
    __shared__ double sh[kVec / 32];
    double t = 0.0;
    for (int b = threadIdx.x; b < nb; b += kVec) t += part[b];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = t;
    __syncthreads();
    t = 0.0;
    for (int q = 0; q < kVec / 32; q++) t += sh[q];
    const double d = ::sqrt(t), f = d > 0.0 ? 1.0 / d : 0.0;
    if (blockIdx.x == 0 && threadIdx.x == 0) *s = d;
    for (size_t i = blockIdx.x * (size_t)kVec + threadIdx.x; i < n; i += (size_t)gridDim.x * kVec) {
        const double v = f * x[i];
        y[i] = v;
        if (z) z[i] = v;
    }
}

__global__ void __launch_bounds__(kVec) k_scale_copy(double* __restrict__ y, const double* __restrict__ x, double s, size_t n)
{
    for (size_t i = blockIdx.x * (size_t)kVec + threadIdx.x; i < n; i += (size_t)gridDim.x * kVec) y[i] = s * x[i];
}

int vec_grid(size_t n) { return static_cast<int>(std::min<size_t>(4 * kSMs, std::max<size_t>(1, (n + kVec - 1) / kVec))); }

// y += sum_k c_k X_k (rows of stride ldx): the 16-byte form when the layout allows
void launch_axpys(cudaStream_t st, double* y, const double* X, size_t ldx, int nk, const double* c, size_t n)
{
    const bool v2 = n % 2 == 0 && ldx % 2 == 0 && reinterpret_cast<uintptr_t>(y) % 16 == 0 &&
        reinterpret_cast<uintptr_t>(X) % 16 == 0;
    if (v2) k_axpys2<<<vec_grid(n / 2), kVec, 0, st>>>(y, X, ldx, nk, c, n);
    else k_axpys<<<vec_grid(n), kVec, 0, st>>>(y, X, ldx, nk, c, n);
}

}  // namespace

struct AdjointWS {
    size_t n = 0;
    int restart = 0;
    double *V = nullptr, *Z = nullptr;  // Krylov basis and preconditioned basis, (restart + 1) x n
    double *w = nullptr, *x = nullptr, *b = nullptr, *t = nullptr, *u = nullptr, *io = nullptr;
    double *part = nullptr, *coef = nullptr;
    double* hcol = nullptr;    // device: the Hessenberg column being formed
    double* h_hcol = nullptr;  // pinned host copy
    cudaEvent_t got_col = nullptr;  // the column of the iteration is in h_hcol
    MatParams<Dual>* mats = nullptr;
    double* dscale = nullptr;
    std::vector<double> h_part;
};

void free_adjoint(Model& m)
{
    if (!m.aws) return;
    AdjointWS& w = *m.aws;
    for (double** p : { &w.V, &w.Z, &w.w, &w.x, &w.b, &w.t, &w.u, &w.io, &w.part, &w.coef, &w.dscale, &w.hcol })
        dev_free(*p);
    if (w.mats) cudaFree(w.mats);
    if (w.h_hcol) cudaFreeHost(w.h_hcol);
    if (w.got_col) cudaEventDestroy(w.got_col);
    delete m.aws;
    m.aws = nullptr;
}

namespace {

efem_status alloc_aws(Model& m)
{
    const size_t n = 3 * static_cast<size_t>(m.n_free);
    if (m.aws && m.aws->n == n) return EFEM_OK;
    free_adjoint(m);
    m.aws = new AdjointWS();
    AdjointWS& w = *m.aws;
    w.n = n;
    w.restart = kRestart;
    efem_status s;
    const size_t nb = static_cast<size_t>(kRestart + 1) * std::max<size_t>(n, 1);
    if ((s = dev_alloc(&w.V, nb)) != EFEM_OK) return s;
    if ((s = dev_alloc(&w.Z, nb)) != EFEM_OK) return s;
    for (double** p : { &w.w, &w.x, &w.b, &w.t, &w.u, &w.io })
        if ((s = dev_alloc(p, std::max<size_t>(n, 1))) != EFEM_OK) return s;
    if ((s = dev_alloc(&w.part, static_cast<size_t>(kRestart + 1) * kGsBlocks)) != EFEM_OK) return s;
    if ((s = dev_alloc(&w.coef, static_cast<size_t>(kRestart + 1))) != EFEM_OK) return s;
    if ((s = dev_alloc(&w.hcol, static_cast<size_t>(kRestart + 2))) != EFEM_OK) return s;
    EFEM_CUDA(cudaMallocHost(&w.h_hcol, sizeof(double) * (kRestart + 2)));
    EFEM_CUDA(cudaEventCreateWithFlags(&w.got_col, cudaEventDisableTiming));
    if ((s = dev_alloc(&w.dscale, static_cast<size_t>(std::max(m.n_pressure_loads, 1)))) != EFEM_OK) return s;
    EFEM_CUDA(cudaMalloc(&w.mats, sizeof(MatParams<Dual>) * MAX_MATS));
    w.h_part.resize(static_cast<size_t>(kRestart + 1) * kDotBlocks);
    return EFEM_OK;
}

// material table on dual numbers; seed (slot, k) puts derivative 1 on constant
// k (0 C10, 1 C01, 2 C20, 3 C30, 4 D1) of material slot `slot`
efem_status upload_dual_mats(Model& m, int slot, int k)
{
    std::vector<MatParams<Dual>> h(std::max<size_t>(m.materials_used.size(), 1));
    for (size_t i = 0; i < m.materials_used.size(); i++) {
        const HostMaterial& hm = m.materials_used[i];
        const bool s = static_cast<int>(i) == slot;
        h[i].type = hm.type;
        h[i].C10 = Dual(hm.C10, s && k == 0 ? 1.0 : 0.0);
        h[i].C01 = Dual(hm.C01, s && k == 1 ? 1.0 : 0.0);
        h[i].C20 = Dual(hm.C20, s && k == 2 ? 1.0 : 0.0);
        h[i].C30 = Dual(hm.C30, s && k == 3 ? 1.0 : 0.0);
        h[i].D1 = Dual(hm.D1, s && k == 4 ? 1.0 : 0.0);
    }
    EFEM_CUDA(cudaMemcpyAsync(m.aws->mats, h.data(), sizeof(MatParams<Dual>) * h.size(), cudaMemcpyHostToDevice, m.stream));
    return EFEM_OK;
}

// out += dR/dtheta of the elements (dual numbers, the seed in the material table)
void launch_elem_param(Model& m, const double* u, double* out)
{
    for (auto& b : m.blocks) {
        if (b.n == 0) continue;
        TanElemArgs a { b.n, m.n_free, b.conn, b.mat, b.vol, b.J0inv, b.dN, b.gw, m.aws->mats, u, nullptr, out };
        const int epb = tan_epb(b.ngp), grid = (b.n + epb - 1) / epb;
        m.launches++;
        if (b.nen == 4 && b.ngp == 1) k_elem_tangent<4, 1><<<grid, kBlock, 0, m.stream>>>(a);
        else if (b.nen == 10 && b.ngp == 4) k_elem_tangent<10, 4><<<grid, kBlock, 0, m.stream>>>(a);
        else if (b.nen == 10 && b.ngp == 1) k_elem_tangent<10, 1><<<grid, kBlock, 0, m.stream>>>(a);
        else if (b.nen == 8 && b.ngp == 8) k_elem_tangent<8, 8><<<grid, kBlock, 0, m.stream>>>(a);
        else if (b.nen == 8 && b.ngp == 1) k_elem_tangent<8, 1><<<grid, kBlock, 0, m.stream>>>(a);
        else if (b.nen == 20 && b.ngp == 27) k_elem_tangent<20, 27><<<grid, kBlock, 0, m.stream>>>(a);
        else if (b.nen == 20 && b.ngp == 8) k_elem_tangent<20, 8><<<grid, kBlock, 0, m.stream>>>(a);
    }
}

TanFaceArgs tan_face_args(const Model& m, const DevFaces& f, const double* u, const double* v, const double* dscale,
    double* out)
{
    return TanFaceArgs { f.n, m.n_free, *std::max_element(f.h_ngp.begin(), f.h_ngp.end()), f.conn, f.table, f.load_idx,
        f.A0, f.J0inv, f.load, f.t_ngp, f.t_w, f.t_N, f.t_dN, u, v, dscale, out };
}

// out -= dF/dscale
void launch_face_param(Model& m, const double* u, const double* dscale, double* out)
{
    for (auto& f : m.faces) {
        if (f.n == 0) continue;
        const TanFaceArgs a = tan_face_args(m, f, u, nullptr, dscale, out);
        const int grid = (f.n + kBlock - 1) / kBlock;
        m.launches++;
        switch (f.nen) {
        case 4: k_face_tangent<4><<<grid, kBlock, 0, m.stream>>>(a); break;
        case 8: k_face_tangent<8><<<grid, kBlock, 0, m.stream>>>(a); break;
        case 10: k_face_tangent<10><<<grid, kBlock, 0, m.stream>>>(a); break;
        case 20: k_face_tangent<20><<<grid, kBlock, 0, m.stream>>>(a); break;
        }
    }
}

// out += K v (transpose: K^T v): every element block's launch carries the faces of its kind
void launch_tangent(Model& m, const double* u, const double* v, double* out, bool transpose)
{
    std::vector<char> done(m.faces.size(), 0);
    for (auto& b : m.blocks) {
        if (b.n == 0) continue;
        TanElemArgs a { b.n, m.n_free, b.conn, b.mat, b.vol, b.J0inv, b.dN, b.gw, nullptr, u, v, out };
        TanFaceArgs fa {};
        int ft = 0;
        for (size_t fs = 0; fs < m.faces.size(); fs++)
            if (!done[fs] && m.faces[fs].n > 0 && m.faces[fs].nen == b.nen) {
                fa = tan_face_args(m, m.faces[fs], u, v, nullptr, out);
                ft = (fa.n + face_epb(b.nen) - 1) / face_epb(b.nen);
                done[fs] = 1;
            }
        const int epb = tan_epb(b.ngp), grid = ft + (b.n + epb - 1) / epb;
        m.launches++;
        auto go = [&](auto nh, auto mr, auto yeoh, auto any) {
            auto* k = b.mat_type == EFEM_NEO_HOOKEAN ? nh : b.mat_type == EFEM_MOONEY_RIVLIN ? mr : b.mat_type == EFEM_YEOH ? yeoh : any;
            k<<<grid, kBlock, 0, m.stream>>>(a, m.d_mats, fa, ft, transpose ? 1 : 0);
        };
#define EFEM_TAN(NEN, NGP)                                                                              \
    if (b.nen == NEN && b.ngp == NGP)                                                                   \
        go(k_tangent<NEN, NGP, EFEM_NEO_HOOKEAN>, k_tangent<NEN, NGP, EFEM_MOONEY_RIVLIN>,              \
            k_tangent<NEN, NGP, EFEM_YEOH>, k_tangent<NEN, NGP, -1>);
        EFEM_TAN(4, 1)
        EFEM_TAN(10, 4)
        EFEM_TAN(10, 1)
        EFEM_TAN(8, 8)
        EFEM_TAN(8, 1)
        EFEM_TAN(20, 27)
        EFEM_TAN(20, 8)
#undef EFEM_TAN
    }
    for (size_t fs = 0; fs < m.faces.size(); fs++) {
        const DevFaces& f = m.faces[fs];
        if (done[fs] || f.n == 0) continue;
        const TanFaceArgs a = tan_face_args(m, f, u, v, nullptr, out);
        const int grid = (f.n + face_epb(f.nen) - 1) / face_epb(f.nen), tr = transpose ? 1 : 0;
        m.launches++;
        switch (f.nen) {
        case 4: k_tangent_faces<4><<<grid, kBlock, 0, m.stream>>>(a, tr); break;
        case 8: k_tangent_faces<8><<<grid, kBlock, 0, m.stream>>>(a, tr); break;
        case 10: k_tangent_faces<10><<<grid, kBlock, 0, m.stream>>>(a, tr); break;
        case 20: k_tangent_faces<20><<<grid, kBlock, 0, m.stream>>>(a, tr); break;
        }
    }
}

// out = K(u) v  (transpose: K(u)^T v); device pointers
efem_status tangent(Model& m, const double* u, const double* v, double* out, bool transpose)
{
    EFEM_CUDA(cudaMemsetAsync(out, 0, sizeof(double) * 3 * m.n_free, m.stream));
    launch_tangent(m, u, v, out, transpose);
    EFEM_CUDA(cudaGetLastError());
    return EFEM_OK;
}

// out = dR/dtheta_k at u (parameter order in the file comment)
efem_status param_derivative(Model& m, const double* u, int k, double* out)
{
    const int nm = static_cast<int>(m.materials_used.size());
    EFEM_CUDA(cudaMemsetAsync(out, 0, sizeof(double) * 3 * m.n_free, m.stream));
    if (k < 5 * nm) {
        efem_status s = upload_dual_mats(m, k / 5, k % 5);
        if (s != EFEM_OK) return s;
        launch_elem_param(m, u, out);
    } else {
        std::vector<double> ds(std::max(m.n_pressure_loads, 1), 0.0);
        ds[k - 5 * nm] = 1.0;
        EFEM_CUDA(cudaMemcpyAsync(m.aws->dscale, ds.data(), sizeof(double) * ds.size(), cudaMemcpyHostToDevice, m.stream));
        launch_face_param(m, u, m.aws->dscale, out);
        // synchronise before ds goes out of scope
        EFEM_CUDA(cudaStreamSynchronize(m.stream));
    }
    EFEM_CUDA(cudaGetLastError());
    return EFEM_OK;
}

// dot products X_k . y for k < nk (X rows of stride n), summed on the host in CTA order
efem_status dots(Model& m, const double* X, int nk, const double* y, double* res)
{
    AdjointWS& w = *m.aws;
    const size_t n = w.n;
    k_dots<<<dim3(kDotBlocks, (nk + kDotRows - 1) / kDotRows), kVec, 0, m.stream>>>(X, n, nk, y, n, w.part);
    m.launches++;
    EFEM_CUDA(cudaMemcpyAsync(w.h_part.data(), w.part, sizeof(double) * nk * kDotBlocks, cudaMemcpyDeviceToHost, m.stream));
    EFEM_CUDA(cudaStreamSynchronize(m.stream));
    for (int k = 0; k < nk; k++) {
        double s = 0.0;
        for (int b = 0; b < kDotBlocks; b++) s += w.h_part[static_cast<size_t>(k) * kDotBlocks + b];
        res[k] = s;
    }
    return EFEM_OK;
}

efem_status axpys(Model& m, double* y, const double* X, int nk, const double* c)
{
    AdjointWS& w = *m.aws;
    EFEM_CUDA(cudaMemcpyAsync(w.coef, c, sizeof(double) * nk, cudaMemcpyHostToDevice, m.stream));
    launch_axpys(m.stream, y, X, w.n, nk, w.coef, w.n);
    m.launches++;
    EFEM_CUDA(cudaStreamSynchronize(m.stream));  // c is host memory owned by the caller
    return EFEM_OK;
}

// Restarted GMRES(kRestart) for K(u)^T x = b, right-preconditioned with H0
// (x = H0 z); classical Gram-Schmidt applied twice.  x starts at 0.
efem_status adjoint_gmres(Model& m, const double* u, double tol, int max_it, int* iters, double* relres,
    double* bytes)
{
    AdjointWS& w = *m.aws;
    const size_t n = w.n;
    const int R = w.restart;
    // algorithmic bytes of one Krylov iteration: the basis copy, H0, the
    // transpose tangent (an FP64 residual plus v and the zeroed output), the
    // norm and the scaling; plus
    // two Gram-Schmidt passes over the j + 1 basis vectors (dots: the basis and
    // w; updates: the basis, w read and written)
    const double nd = 8.0 * static_cast<double>(n);
    efem_model_info mi {};
    precond_info(m, &mi);
    long long rb = 0;
    double rf = 0.0;
    residual_work(m, 8, &rb, &rf, true);
    const double it_bytes = 2.0 * nd + 16.0 * static_cast<double>(mi.factor_nnz) + 5.0 * nd + static_cast<double>(rb) +
        2.0 * nd + 3.0 * nd;
    *bytes = 0.0;
    double bnorm = 0.0;
    efem_status s = dots(m, w.b, 1, w.b, &bnorm);
    if (s != EFEM_OK) return s;
    bnorm = std::sqrt(bnorm);
    EFEM_CUDA(cudaMemsetAsync(w.x, 0, sizeof(double) * n, m.stream));
    *iters = 0;
    *relres = 0.0;
    if (bnorm == 0.0) return EFEM_OK;
    std::vector<double> H(static_cast<size_t>(R + 1) * R), cs(R), sn(R), g(R + 1), y(R);
    double beta = bnorm;  // residual of x = 0
    EFEM_CUDA(cudaMemcpyAsync(w.t, w.b, sizeof(double) * n, cudaMemcpyDeviceToDevice, m.stream));
    int total = 0;
    while (total < max_it) {
        // V_0 = r / beta, r = t, and its copy for H0
        k_scale_copy<<<vec_grid(n), kVec, 0, m.stream>>>(w.V, w.t, 1.0 / beta, n);
        k_scale_copy<<<vec_grid(n), kVec, 0, m.stream>>>(w.Z, w.t, 1.0 / beta, n);
        m.launches += 2;
        std::fill(g.begin(), g.end(), 0.0);
        g[0] = beta;
        int j = 0;
        bool done = false;
        // w.w = K^T H0 V_j (Z_j: the copy of V_j, then H0 V_j)
        auto product = [&](int jj) -> efem_status {
            efem_status ps = precond_enqueue(m, w.Z + jj * n, m.stream);
            if (ps != EFEM_OK) return ps;
            m.launches += precond_launch_count(m);
            return tangent(m, u, w.Z + jj * n, w.w, true);
        };
        if ((s = product(0)) != EFEM_OK) return s;
        for (; j < R && total < max_it; j++, total++) {
            *bytes += it_bytes + 2.0 * (2.0 * (j + 1) * nd + 3.0 * nd);
            // two passes of classical Gram-Schmidt, coefficients kept on the device
            // (with H0 a good preconditioner, K^T H0 v is close to the basis: the
            // first pass removes most of w in nearly every iteration, so a
            // conditional second pass would almost always run)
            k_dots<<<dim3(kDotBlocks, (j + kDotRows) / kDotRows), kVec, 0, m.stream>>>(w.V, n, j + 1, w.w, n, w.part);
            k_rows_reduce<<<(j + 1 + 7) / 8, 256, 0, m.stream>>>(w.part, j + 1, kDotBlocks, w.hcol, w.coef, 0);
            k_gs_update<false><<<kGsBlocks, kVec, 0, m.stream>>>(w.w, w.V, n, j + 1, w.coef, n, w.part);
            k_rows_reduce<<<(j + 1 + 7) / 8, 256, 0, m.stream>>>(w.part, j + 1, kGsBlocks, w.hcol, w.coef, 1);
            k_gs_update<true><<<kGsNormBlocks, kVec, 0, m.stream>>>(w.w, w.V, n, j + 1, w.coef, n, w.part);
            k_gs_scale<<<vec_grid(n), kVec, 0, m.stream>>>(w.V + (j + 1) * n, j + 1 < R ? w.Z + (j + 1) * n : nullptr, w.w,
                w.part, kGsNormBlocks, w.hcol + j + 1, n);
            m.launches += 6;
            EFEM_CUDA(cudaMemcpyAsync(w.h_hcol, w.hcol, sizeof(double) * (j + 2), cudaMemcpyDeviceToHost, m.stream));
            EFEM_CUDA(cudaEventRecord(w.got_col, m.stream));
            // the next iteration's product starts while the host reads the column
            // (one product too many when this iteration converges)
            if (j + 1 < R && total + 1 < max_it && (s = product(j + 1)) != EFEM_OK) return s;
            EFEM_CUDA(cudaEventSynchronize(w.got_col));
            for (int i = 0; i <= j + 1; i++) H[static_cast<size_t>(i) * R + j] = w.h_hcol[i];
            const double hn = w.h_hcol[j + 1];
            // Givens rotations on column j
            for (int i = 0; i < j; i++) {
                const double a = H[static_cast<size_t>(i) * R + j], c = H[static_cast<size_t>(i + 1) * R + j];
                H[static_cast<size_t>(i) * R + j] = cs[i] * a + sn[i] * c;
                H[static_cast<size_t>(i + 1) * R + j] = -sn[i] * a + cs[i] * c;
            }
            const double a = H[static_cast<size_t>(j) * R + j], c = H[static_cast<size_t>(j + 1) * R + j];
            const double rr = std::hypot(a, c);
            cs[j] = rr > 0.0 ? a / rr : 1.0;
            sn[j] = rr > 0.0 ? c / rr : 0.0;
            H[static_cast<size_t>(j) * R + j] = rr;
            H[static_cast<size_t>(j + 1) * R + j] = 0.0;
            g[j + 1] = -sn[j] * g[j];
            g[j] = cs[j] * g[j];
            *relres = std::fabs(g[j + 1]) / bnorm;
            // not finite (an H0 application that gave up leaves NaN, or u or dJ/du
            // hold one): nothing that follows could become finite again
            if (*relres <= tol || hn == 0.0 || !std::isfinite(*relres) || !std::isfinite(hn)) {
                j++;
                total++;
                done = true;
                break;
            }
        }
        // x += Z y, H y = g (upper triangular j x j)
        for (int i = j - 1; i >= 0; i--) {
            double t = g[i];
            for (int k = i + 1; k < j; k++) t -= H[static_cast<size_t>(i) * R + k] * y[k];
            y[i] = t / H[static_cast<size_t>(i) * R + i];
        }
        if ((s = axpys(m, w.x, w.Z, j, y.data())) != EFEM_OK) return s;
        if ((s = precond_check(m)) != EFEM_OK) return s;
        if (done) break;
        // true residual t = b - K^T x for the restart
        if ((s = tangent(m, u, w.x, w.w, true)) != EFEM_OK) return s;
        k_scale_copy<<<vec_grid(n), kVec, 0, m.stream>>>(w.t, w.b, 1.0, n);
        m.launches++;
        const double minus1 = -1.0;
        if ((s = axpys(m, w.t, w.w, 1, &minus1)) != EFEM_OK) return s;
        if ((s = dots(m, w.t, 1, w.t, &beta)) != EFEM_OK) return s;
        beta = std::sqrt(beta);
        *relres = beta / bnorm;
        if (*relres <= tol) break;
    }
    *iters = total;
    return EFEM_OK;
}

double ms_since(std::chrono::steady_clock::time_point t0)
{
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

}  // namespace

// ------------------------------------------------------------------ host entry points (C ABI helpers)
efem_status adjoint_io(Model& m, double** io)
{
    efem_status s = alloc_aws(m);
    if (s != EFEM_OK) return s;
    *io = m.aws->io;
    return EFEM_OK;
}

int n_params(const Model& m) { return 5 * static_cast<int>(m.materials_used.size()) + m.n_pressure_loads; }

efem_status hvp(Model& m, const double* d_u, const double* d_v, double* d_out, bool transpose)
{
    efem_status s = alloc_aws(m);
    if (s != EFEM_OK) return s;
    return tangent(m, d_u, d_v, d_out, transpose);
}

efem_status residual_param_derivative(Model& m, const double* d_u, int k, double* d_out)
{
    if (k < 0 || k >= n_params(m)) {
        set_error("parameter index out of range");
        return EFEM_ERR_ARG;
    }
    efem_status s = alloc_aws(m);
    if (s != EFEM_OK) return s;
    return param_derivative(m, d_u, k, d_out);
}

efem_status adjoint(Model& m, const double* d_u, const double* d_dJdu, double* dJdtheta, double* d_lambda,
    efem_adjoint_info* info)
{
    const auto t0 = std::chrono::steady_clock::now();
    std::memset(info, 0, sizeof(*info));
    const long long launches0 = m.launches;
    efem_status s = alloc_aws(m);
    if (s != EFEM_OK) return s;
    AdjointWS& w = *m.aws;
    const size_t n = w.n;
    int ok = 0;
    double msf = 0.0;
    if ((s = precond_setup(m, false, &ok, &msf)) != EFEM_OK) return s;
    if (!ok) {
        set_error("approximate Jacobian is not positive definite (no preconditioner for the adjoint solve)");
        return EFEM_ERR_NAN;
    }
    EFEM_CUDA(cudaMemcpyAsync(w.u, d_u, sizeof(double) * n, cudaMemcpyDeviceToDevice, m.stream));
    EFEM_CUDA(cudaMemcpyAsync(w.b, d_dJdu, sizeof(double) * n, cudaMemcpyDeviceToDevice, m.stream));
    const double tol = m.opts.adjoint_tolerance > 0 ? m.opts.adjoint_tolerance : 1e-8;
    const int max_it = m.opts.adjoint_max_iterations > 0 ? m.opts.adjoint_max_iterations : 2000;
    int iters = 0;
    double rel = 0.0;
    s = adjoint_gmres(m, w.u, tol, max_it, &iters, &rel, &info->solve_bytes);
    if (s != EFEM_OK) return s;
    info->iterations = iters;
    info->rel_residual = rel;
    if (rel <= tol) info->flags |= EFEM_SOLVE_CONVERGED;
    EFEM_CUDA(cudaStreamSynchronize(m.stream));
    info->ms_solve = ms_since(t0);
    // dJ/dtheta_k = -lambda . dR/dtheta_k
    const auto t1 = std::chrono::steady_clock::now();
    const int np = n_params(m);
    for (int k = 0; k < np; k++) {
        if ((s = param_derivative(m, w.u, k, w.t)) != EFEM_OK) return s;
        double d = 0.0;
        if ((s = dots(m, w.t, 1, w.x, &d)) != EFEM_OK) return s;
        dJdtheta[k] = -d;
    }
    if (d_lambda) EFEM_CUDA(cudaMemcpyAsync(d_lambda, w.x, sizeof(double) * n, cudaMemcpyDeviceToDevice, m.stream));
    EFEM_CUDA(cudaStreamSynchronize(m.stream));
    info->ms_params = ms_since(t1);
    info->ms_total = ms_since(t0);
    info->n_kernel_launches = m.launches - launches0;
    return EFEM_OK;
}

}  // namespace efem
