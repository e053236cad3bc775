// Residual R(u) = f_int(u) - f_ext(u) on the GPU.
//
//   element internal force   r_e = V_e sum_g w_g P(F_g) T_g
//                            (src/fe/ElementConstraint.cpp:139-162)
//   follower pressure        f_i = p sum_g w_g N_i(xi_g) cof(F_g) A0, r_i -= f_i
//   directed pressure        f_i = v sum_g w_g N_i(xi_g) |cof(F_g) A0|
//                            (src/fe/ExternalConstraint.cpp:829-959)
//   nodal forces             r starts from -f_ext (:149-167)
//
// Element kernel (k_elem_thread replaces it for FP32 C3D20 with 27 points where
// it is faster): one CTA processes EPB elements in three phases.
//   1. stage: threads (element, node) load conn (SoA, coalesced over elements)
//      and gather u, relative to the element's first node, into shared memory;
//   2. Gauss point: thread (element, gp) forms H = (u . dN) J0^{-1}, P(I+H) and
//      S_g = V_e w_g P J0^{-T} (3x3) into shared memory;
//   3. node: thread (element, node) reduces r_a = sum_g S_g dN_ga and adds it
//      to the global residual with FP64 atomics (red.global.add.f64) or, in
//      deterministic mode (opts.deterministic), stores it in its own slot of a
//      contribution buffer that k_gather then sums per node in ascending slot
//      order, so the residual is bitwise repeatable.
// The arithmetic type T is double (FP64 path) or float (mixed path); the
// global residual is always accumulated in FP64.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <type_traits>
#include <vector>

#include "efem_internal.h"
#include "mechanics.cuh"

namespace efem {

namespace {

constexpr int kBlock = 128;

template <typename T>
struct ElemArgs {
    int n, n_free;
    const int* __restrict__ conn;     // [NEN][n]
    const int* __restrict__ mat;      // [n]
    const T* __restrict__ vol;        // [n]
    const T* __restrict__ J0inv;      // [n][NGP][9]
    const T* __restrict__ dN;         // [NGP][NEN][3]
    const T* __restrict__ gw;         // [NGP]
    const MatParams<T>* __restrict__ mats;
    const double* __restrict__ u;     // [3*n_free]
    double* __restrict__ r;           // [3*n_free]
    double* __restrict__ contrib;     // deterministic scatter: [3][n_slots], or null for atomics
    size_t n_slots, slot0;
    const int* __restrict__ egroup;   // batch unions: the member of every element
    const int* frozen;                // batch unions: 1 for a member that no longer iterates (null: none)
};

// where an (element or face, node) pair's nodal force goes
struct Scatter {
    double* contrib = nullptr;
    size_t n_slots = 0, slot0 = 0;
};

// BLK threads per CTA (64, 128 or 256, picked per element block by the
// autotuner in tune_element_blocks); EPB = BLK / NGP elements per CTA, at
// most 128 (shared memory)
template <int NGP, int BLK>
constexpr int elems_per_cta() { return (BLK / NGP) < 1 ? 1 : ((BLK / NGP) > 128 ? 128 : BLK / NGP); }

template <typename T>
struct FaceArgs {
    int n, n_free;
    int gmax;                         // most points of a face in the set
    const int* __restrict__ conn;     // [NEN][n]
    const int* __restrict__ table;    // [n]
    const double* __restrict__ A0;    // [n][3]
    const T* __restrict__ J0inv;      // [n][MAX_FGP][9]
    const double* __restrict__ load;  // [n][4]
    const int* __restrict__ t_ngp;
    const T* __restrict__ t_w;        // [t][MAX_FGP]
    const T* __restrict__ t_N;        // [t][MAX_FGP][NEN]
    const T* __restrict__ t_dN;       // [t][MAX_FGP][NEN][3]
    const double* __restrict__ u;
    double* __restrict__ r;
    double* __restrict__ contrib;     // deterministic scatter: [3][n_slots], or null for atomics
    size_t n_slots, slot0;
};

// Pressure faces, EPB per tile, in the element kernel's phases: (face, node)
// threads stage u, (face, point) threads form cof(F_g) A0, and (face, node)
// threads add up and scatter the nodal forces.  A face is a few hundred
// dependent FP64 operations, so latency bounds it and not its work: with one
// thread per face, all in that thread's local memory, the 2 752 faces of the
// C3D20R cap took 34.8 us (22 CTAs), more than twice its elements; in phases
// 11.4 us by themselves.  The element kernel's launch carries them as its
// first CTAs (k_elem_residual), where they overlap with the elements.
template <int NEN, int BLK>
constexpr int face_epb() { return (NEN >= 20 ? 8 : NEN >= 8 ? 16 : 32) * BLK / 128; }

template <int NEN, typename T, int EPB>
struct FaceSmem {
    T u[EPB][(NEN * 3) | 1];       // displacements relative to the parent's first node, as in the element kernel
    T cA[EPB][(MAX_FGP * 3) | 1];  // cof(F_g) A0 (directed loads: its norm) at every face point
    int node[EPB][NEN];
    int table[EPB], ngp[EPB];
};

template <int NEN, typename T, int BLK>
__device__ void face_tile(const FaceArgs<T>& a, int tile, FaceSmem<NEN, T, face_epb<NEN, BLK>()>& sm)
{
    constexpr int EPB = face_epb<NEN, BLK>();
    const int tid = threadIdx.x, fb = tile * EPB;
    // the (face, point) pair of phase 2: its inputs are on their way while u is staged
    const int el1 = tid / a.gmax, g1 = tid - el1 * a.gmax, f1 = fb + el1;
    const bool on1 = tid < EPB * a.gmax && f1 < a.n;
    T Ji1[9], A01[3];
#pragma unroll
    for (int k = 0; k < 9; k++) Ji1[k] = on1 ? __ldg(a.J0inv + (static_cast<size_t>(f1) * MAX_FGP + g1) * 9 + k) : T(0);
#pragma unroll
    for (int k = 0; k < 3; k++) A01[k] = on1 ? static_cast<T>(__ldg(a.A0 + 3 * f1 + k)) : T(0);
    const double directed1 = on1 ? __ldg(a.load + 4 * f1) : 0.0;
    if (tid < EPB) {
        const int t = fb + tid < a.n ? __ldg(a.table + fb + tid) : 0;
        sm.table[tid] = t;
        sm.ngp[tid] = __ldg(a.t_ngp + t);
    }
    for (int i = tid; i < EPB * NEN; i += BLK) {
        const int el = i % EPB, q = i / EPB, f = fb + el;
        int node = a.n_free;
        double u0 = 0.0, u1 = 0.0, u2 = 0.0;
        if (f < a.n) {
            node = __ldg(a.conn + static_cast<size_t>(q) * a.n + f);
            const int n0 = __ldg(a.conn + f);
            double z0 = 0.0, z1 = 0.0, z2 = 0.0;
            if (node < a.n_free) {
                u0 = __ldg(a.u + 3 * node);
                u1 = __ldg(a.u + 3 * node + 1);
                u2 = __ldg(a.u + 3 * node + 2);
            }
            if (n0 < a.n_free) {
                z0 = __ldg(a.u + 3 * n0);
                z1 = __ldg(a.u + 3 * n0 + 1);
                z2 = __ldg(a.u + 3 * n0 + 2);
            }
            u0 -= z0;
            u1 -= z1;
            u2 -= z2;
        }
        sm.node[el][q] = node;
        sm.u[el][3 * q] = static_cast<T>(u0);
        sm.u[el][3 * q + 1] = static_cast<T>(u1);
        sm.u[el][3 * q + 2] = static_cast<T>(u2);
    }
    __syncthreads();
    for (int i = tid; i < EPB * a.gmax; i += BLK) {
        const int el = i / a.gmax, g = i - el * a.gmax, f = fb + el;
        if (f >= a.n) break;
        if (g >= sm.ngp[el]) continue;
        const T* dN = a.t_dN + (static_cast<size_t>(sm.table[el]) * MAX_FGP + g) * NEN * 3;
        T Ji[9], A0[3];
        double directed = directed1;
#pragma unroll
        for (int k = 0; k < 9; k++) Ji[k] = Ji1[k];
#pragma unroll
        for (int k = 0; k < 3; k++) A0[k] = A01[k];
        if (i != tid) {  // more (face, point) pairs than threads
#pragma unroll
            for (int k = 0; k < 9; k++) Ji[k] = __ldg(a.J0inv + (static_cast<size_t>(f) * MAX_FGP + g) * 9 + k);
#pragma unroll
            for (int k = 0; k < 3; k++) A0[k] = static_cast<T>(__ldg(a.A0 + 3 * f + k));
            directed = __ldg(a.load + 4 * f);
        }
        T A[9] = { 0, 0, 0, 0, 0, 0, 0, 0, 0 };
#pragma unroll(NEN == 4 ? 4 : 5)
        for (int q = 0; q < NEN; q++)
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int k = 0; k < 3; k++) A[3 * c + k] += sm.u[el][3 * q + c] * __ldg(dN + 3 * q + k);
        T H[9];
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
            for (int j = 0; j < 3; j++) H[3 * c + j] = A[3 * c] * Ji[j] + A[3 * c + 1] * Ji[3 + j] + A[3 * c + 2] * Ji[6 + j];
        Kin<T> k;
        kinematics(H, k);
        // cof F A0 = (I + B) A0
        T cA[3];
#pragma unroll
        for (int c = 0; c < 3; c++) cA[c] = A0[c] + k.B[3 * c] * A0[0] + k.B[3 * c + 1] * A0[1] + k.B[3 * c + 2] * A0[2];
        if (directed != 0.0) cA[0] = sqrt(cA[0] * cA[0] + cA[1] * cA[1] + cA[2] * cA[2]);
#pragma unroll
        for (int c = 0; c < 3; c++) sm.cA[el][3 * g + c] = cA[c];
    }
    __syncthreads();
    for (int i = tid; i < EPB * NEN; i += BLK) {
        const int el = i % EPB, q = i / EPB, f = fb + el;
        if (f >= a.n) continue;
        const int node = sm.node[el][q];
        if (node >= a.n_free) continue;
        const int t = sm.table[el], ngp = sm.ngp[el];
        const T* tw = a.t_w + t * MAX_FGP;
        const T* tN = a.t_N + static_cast<size_t>(t) * MAX_FGP * NEN + q;
        const double* L = a.load + 4 * f;
        const double l0 = __ldg(L), l1 = __ldg(L + 1), l2 = __ldg(L + 2), l3 = __ldg(L + 3);
        T v0 = 0, v1 = 0, v2 = 0;
#pragma unroll 3
        for (int g = 0; g < ngp; g++) {
            const T wn = __ldg(tw + g) * __ldg(tN + g * NEN);
            v0 += wn * sm.cA[el][3 * g];
            v1 += wn * sm.cA[el][3 * g + 1];
            v2 += wn * sm.cA[el][3 * g + 2];
        }
        double f0, f1, f2;
        if (l0 != 0.0) {
            f0 = l1 * static_cast<double>(v0);
            f1 = l2 * static_cast<double>(v0);
            f2 = l3 * static_cast<double>(v0);
        } else {
            f0 = l1 * static_cast<double>(v0);
            f1 = l1 * static_cast<double>(v1);
            f2 = l1 * static_cast<double>(v2);
        }
        if (a.contrib) {
            const size_t sl = a.slot0 + static_cast<size_t>(q) * a.n + f;
            a.contrib[sl] = -f0;
            a.contrib[a.n_slots + sl] = -f1;
            a.contrib[2 * a.n_slots + sl] = -f2;
        } else {
            atomicAdd(a.r + 3 * node, -f0);
            atomicAdd(a.r + 3 * node + 1, -f1);
            atomicAdd(a.r + 3 * node + 2, -f2);
        }
    }
}

// faces without an element block of their kind to go with
template <int NEN, typename T>
__global__ void __launch_bounds__(kBlock) k_face_residual(FaceArgs<T> a)
{
    griddep_wait();
    __shared__ FaceSmem<NEN, T, face_epb<NEN, kBlock>()> sm;
    face_tile<NEN, T, kBlock>(a, blockIdx.x, sm);
    griddep_launch();
}

template <int NEN, int NGP, typename T, int EPB>
struct ElemSmem {
    // per-element rows padded to an odd length, so that threads on
    // consecutive elements (phases 1 and 3) or Gauss points (phase 2) read
    // different shared-memory banks
    T u[EPB][(NEN * 3) | 1];   // [element][node * 3 + component]
    T S[EPB][(NGP * 9) | 1];   // [element][gp * 9 + 3 i + j]
    T dN[NGP][(NEN * 3) | 1];  // [gp][node * 3 + k]
    int node[EPB][NEN | 1];
};

struct NoFaces {};
template <int NEN, typename T, int BLK, bool Faces>
using FaceSmemIf = std::conditional_t<Faces, FaceSmem<NEN, T, face_epb<NEN, BLK>()>, NoFaces>;

// MT: the block's one material law, or -1 when its elements mix laws.  With
// Faces the first n_face_tiles CTAs take the pressure faces of the block's
// kind.  Blocks without faces have a kernel without them: a kernel's registers
// are the larger of the two parts', and the faces' cost the neo-Hookean FP64
// elements a third of their warps (C3D8 64 -> 92 registers; the residual of
// 119 700 elements 53.0 -> 57.0 us, of 105 000 C3D10 tetrahedra 37.5 -> 39.7).
// With faces the one launch is the faster one all the same (57.5 against 64.9
// and 40.3 against 49.5 us for two).
template <int NEN, int NGP, typename T, int BLK, int MT, bool Faces>
__global__ void __launch_bounds__(BLK) k_elem_residual(ElemArgs<T> a, FaceArgs<T> fa, int n_face_tiles)
{
    griddep_wait();
    constexpr int EPB = elems_per_cta<NGP, BLK>();
    __shared__ union Smem {
        ElemSmem<NEN, NGP, T, EPB> e;
        FaceSmemIf<NEN, T, BLK, Faces> f;
        __device__ Smem() {}
    } smem;
    if constexpr (Faces) {
        if (static_cast<int>(blockIdx.x) < n_face_tiles) {
            face_tile<NEN, T, BLK>(fa, blockIdx.x, smem.f);
            griddep_launch();
            return;
        }
    }
    auto& s_u = smem.e.u;
    auto& s_S = smem.e.S;
    auto& s_dN = smem.e.dN;
    auto& s_node = smem.e.node;

    const int tid = threadIdx.x;
    const int e0 = (static_cast<int>(blockIdx.x) - (Faces ? n_face_tiles : 0)) * EPB;
    if (a.frozen) {  // a batch union: skip the CTA when every member it covers has stopped iterating
        const int e1 = min(a.n, e0 + EPB) - 1;
        bool act = false;
        for (int g = __ldg(a.egroup + e0); g <= __ldg(a.egroup + e1); g++) act = act || !a.frozen[g];
        if (!act) {
            griddep_launch();
            return;
        }
    }
    for (int i = tid; i < NGP * NEN * 3; i += BLK) s_dN[i / (NEN * 3)][i % (NEN * 3)] = a.dN[i];

    // phase 1: stage node displacements relative to the element's first node,
    // formed in FP64 (H only sees differences, since sum_a dN_a = 0, and FP32
    // would lose the differences of nearly equal displacements)
    for (int i = tid; i < EPB * NEN; i += BLK) {
        const int el = i % EPB, nd = i / EPB, e = e0 + el;
        int node = a.n_free;  // out-of-range marker
        T v0 = 0, v1 = 0, v2 = 0;
        if (e < a.n) {
            node = __ldg(a.conn + static_cast<size_t>(nd) * a.n + e);
            const int n0 = __ldg(a.conn + e);
            double w0 = 0.0, w1 = 0.0, w2 = 0.0, z0 = 0.0, z1 = 0.0, z2 = 0.0;
            if (node < a.n_free) {
                w0 = __ldg(a.u + 3 * node);
                w1 = __ldg(a.u + 3 * node + 1);
                w2 = __ldg(a.u + 3 * node + 2);
            }
            if (n0 < a.n_free) {
                z0 = __ldg(a.u + 3 * n0);
                z1 = __ldg(a.u + 3 * n0 + 1);
                z2 = __ldg(a.u + 3 * n0 + 2);
            }
            v0 = static_cast<T>(w0 - z0);
            v1 = static_cast<T>(w1 - z1);
            v2 = static_cast<T>(w2 - z2);
        }
        s_node[el][nd] = node;
        s_u[el][3 * nd] = v0;
        s_u[el][3 * nd + 1] = v1;
        s_u[el][3 * nd + 2] = v2;
    }
    __syncthreads();

    // phase 2: one thread per (element, Gauss point)
    if (tid < EPB * NGP) {
        const int el = tid / NGP, g = tid % NGP, e = e0 + el;
        if (e < a.n) {
            T A[9];
#pragma unroll
            for (int k = 0; k < 9; k++) A[k] = 0;
#pragma unroll 4
            for (int q = 0; q < NEN; q++) {
                const T u0 = s_u[el][3 * q], u1 = s_u[el][3 * q + 1], u2 = s_u[el][3 * q + 2];
                const T d0 = s_dN[g][3 * q], d1 = s_dN[g][3 * q + 1], d2 = s_dN[g][3 * q + 2];
                A[0] += u0 * d0; A[1] += u0 * d1; A[2] += u0 * d2;
                A[3] += u1 * d0; A[4] += u1 * d1; A[5] += u1 * d2;
                A[6] += u2 * d0; A[7] += u2 * d1; A[8] += u2 * d2;
            }
            const T* Jp = a.J0inv + (static_cast<size_t>(e) * NGP + g) * 9;
            T H[9];
            {
                T Ji[9];
#pragma unroll
                for (int k = 0; k < 9; k++) Ji[k] = __ldg(Jp + k);
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int j = 0; j < 3; j++)
                        H[3 * i + j] = A[3 * i] * Ji[j] + A[3 * i + 1] * Ji[3 + j] + A[3 * i + 2] * Ji[6 + j];
            }
            const MatParams<T> mp = a.mats[__ldg(a.mat + e)];
            T P[9];
            piola<T, MT>(mp, H, P);
            const T wv = __ldg(a.vol + e) * a.gw[g];
            // S = wv P J0^{-T}; J0^{-1} read again (an L1 hit) rather than
            // kept in registers through the stress law
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const T j0 = __ldg(Jp + 3 * j), j1 = __ldg(Jp + 3 * j + 1), j2 = __ldg(Jp + 3 * j + 2);
#pragma unroll
                for (int i = 0; i < 3; i++) s_S[el][9 * g + 3 * i + j] = wv * (P[3 * i] * j0 + P[3 * i + 1] * j1 + P[3 * i + 2] * j2);
            }
        }
    }
    __syncthreads();

    // phase 3: one thread per (element, node): r_a = sum_g S_g dN_ga
    for (int i = tid; i < EPB * NEN; i += BLK) {
        const int el = i % EPB, nd = i / EPB, e = e0 + el;
        if (e >= a.n) continue;
        const int node = s_node[el][nd];
        if (node >= a.n_free) continue;
        T r0 = 0, r1 = 0, r2 = 0;
#pragma unroll 4
        for (int g = 0; g < NGP; g++) {
            const T d0 = s_dN[g][3 * nd], d1 = s_dN[g][3 * nd + 1], d2 = s_dN[g][3 * nd + 2];
            const T* S = &s_S[el][9 * g];
            r0 += S[0] * d0 + S[1] * d1 + S[2] * d2;
            r1 += S[3] * d0 + S[4] * d1 + S[5] * d2;
            r2 += S[6] * d0 + S[7] * d1 + S[8] * d2;
        }
        if (a.contrib) {  // consecutive threads: consecutive elements, consecutive slots
            const size_t sl = a.slot0 + static_cast<size_t>(nd) * a.n + e;
            a.contrib[sl] = static_cast<double>(r0);
            a.contrib[a.n_slots + sl] = static_cast<double>(r1);
            a.contrib[2 * a.n_slots + sl] = static_cast<double>(r2);
        } else {
            atomicAdd(a.r + 3 * node, static_cast<double>(r0));
            atomicAdd(a.r + 3 * node + 1, static_cast<double>(r1));
            atomicAdd(a.r + 3 * node + 2, static_cast<double>(r2));
        }
    }
    griddep_launch();
}

// The FP32 kernel of 20 nodes and 27 points: G threads per element, in
// different warps, share its Gauss points.  k_elem_residual reads 6
// shared-memory words per 9 multiply-adds of phase 2 and 12 per 9 of phase 3
// (79% of the memory pipe with 27 points); here a node's u is one 16-byte word
// of the thread's own column, dN a broadcast (every lane of a warp is at the
// same point) and the forces are added up in registers.  J0^{-1} of the next
// point is fetched by the warp for its 32 elements, coalesced, while this one
// is worked on.  What bounds it: issue slots 57% busy and no warp ready in
// the other cycles at 16 warps an SM (8 CTAs by 128 registers, 60 of them sums,
// and by shared memory); and the last wave, for which 7 CTAs an SM are sometimes
// the better number, so the autotuner times both (`pad`).
// One residual in a solve, neo-Hookean, with 8 and 7: 36 864 elements 53 and
// 64 us, 60 625 elements 84 and 82, 70 713 elements 96 and 105.
// A direct call on 60 625 elements went from 131 to 105 us (G = 1: 5 us more).  For 4 to 10 nodes, 8 points of 20, and in FP64,
// where the sums do not fit or are few, k_elem_residual was as fast or faster
// (FP32: C3D8 25.0 against 25.8, C3D10 32.4 against 34.1, C3D20R 28.0 against
// 30.8 us), and small blocks want its many threads: the autotuner decides.
constexpr int kTB = 64;    // threads
constexpr int kSplit = 2;  // threads per element
constexpr int kPerSM = 8;  // CTAs per SM
constexpr size_t kPadSmem = 2048;  // dynamic shared memory that leaves room for 7
constexpr size_t kSmemSM = 233472, kSmemCTA = 1024;  // shared memory of an SM, and what the system takes of it per CTA

template <typename T>
constexpr bool has_thread_kernel(int nen, int ngp) { return sizeof(T) == 4 && nen == 20 && ngp == 27; }

// three values of a row of four
__device__ __forceinline__ void load3(const float* p, float& a, float& b, float& c)
{
    const float4 v = *reinterpret_cast<const float4*>(p);
    a = v.x;
    b = v.y;
    c = v.z;
}

template <int NEN, int NGP, int MT, int G>
__global__ void __launch_bounds__(kTB, kPerSM) k_elem_thread(ElemArgs<float> a, FaceArgs<float> fa, int n_face_tiles)
{
    griddep_wait();
    using T = float;
    constexpr int E = kTB / G;  // elements
    __shared__ union Smem {
        struct {
            alignas(16) T dN[NGP * NEN * 4];
            alignas(16) T w[4 * NEN * E > 3 * NEN * G * E ? 4 * NEN * E : 3 * NEN * G * E];  // u [NEN][E][4]; at the end the sums [G][3 NEN][E]
            T J[kTB / 32][32 * 9];           // a warp's J0^{-1} at its Gauss point
        } e;
        FaceSmem<NEN, T, face_epb<NEN, kTB>()> f;
        __device__ Smem() {}
    } smem;
    static_assert(kPerSM * (sizeof(Smem) + kSmemCTA) <= kSmemSM, "kPerSM CTAs on an SM");
    static_assert(kPerSM * (sizeof(Smem) + kSmemCTA + kPadSmem) > kSmemSM, "one less with the pad");
    if (static_cast<int>(blockIdx.x) < n_face_tiles) {
        face_tile<NEN, T, kTB>(fa, blockIdx.x, smem.f);
        griddep_launch();
        return;
    }
    T* su = smem.e.w;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int part = w % G, grp = w / G, el = grp * 32 + lane;
    const int e0 = (static_cast<int>(blockIdx.x) - n_face_tiles) * E, e = e0 + el, ew = e0 + grp * 32;
    if (a.frozen) {  // a batch union: skip the CTA when every member it covers has stopped iterating
        const int e1 = min(a.n, e0 + E) - 1;
        bool act = false;
        for (int g = __ldg(a.egroup + e0); g <= __ldg(a.egroup + e1); g++) act = act || !a.frozen[g];
        if (!act) {
            griddep_launch();
            return;
        }
    }
    T* sJ = smem.e.J[w];
    T jn[9];
    const T* J0 = a.J0inv + static_cast<size_t>(ew) * NGP * 9;
    const int jmax = min(a.n - ew, 32) * (NGP * 9);
    int jo[9];  // the lane's offsets in the warp's J0^{-1} at point 0 (past jmax: no element)
#pragma unroll
    for (int k = 0; k < 9; k++) jo[k] = (k * 32 + lane) / 9 * (NGP * 9) + (k * 32 + lane) % 9;
    auto fetch = [&](int g) {
#pragma unroll
        for (int k = 0; k < 9; k++) jn[k] = jo[k] < jmax ? __ldg(J0 + jo[k] + g * 9) : T(0);
    };
    fetch(part);
    for (int i = tid; i < NGP * NEN * 3; i += kTB) smem.e.dN[i / 3 * 4 + i % 3] = a.dN[i];
    // displacements relative to the element's first node, formed in FP64 (as in k_elem_residual)
    const int ec = min(e, a.n - 1);
    {
        const int n0 = __ldg(a.conn + ec);
        double z0 = 0.0, z1 = 0.0, z2 = 0.0;
        if (n0 < a.n_free) {
            z0 = __ldg(a.u + 3 * n0);
            z1 = __ldg(a.u + 3 * n0 + 1);
            z2 = __ldg(a.u + 3 * n0 + 2);
        }
#pragma unroll
        for (int q = part; q < NEN; q += G) {
            const int node = __ldg(a.conn + static_cast<size_t>(q) * a.n + ec);
            double w0 = 0.0, w1 = 0.0, w2 = 0.0;
            if (node < a.n_free) {
                w0 = __ldg(a.u + 3 * node);
                w1 = __ldg(a.u + 3 * node + 1);
                w2 = __ldg(a.u + 3 * node + 2);
            }
            *reinterpret_cast<float4*>(su + (q * E + el) * 4)
                = make_float4(static_cast<T>(w0 - z0), static_cast<T>(w1 - z1), static_cast<T>(w2 - z2), 0.0f);
        }
    }
    const MatParams<T>* mp = a.mats + __ldg(a.mat + ec);
    const T vol = __ldg(a.vol + ec);
    T f[3 * NEN];
#pragma unroll
    for (int k = 0; k < 3 * NEN; k++) f[k] = 0;
    __syncthreads();
#pragma unroll 1
    for (int g = part; g < NGP; g += G) {
#pragma unroll
        for (int k = 0; k < 9; k++) sJ[k * 32 + lane] = jn[k];
        __syncwarp();
        if (g + G < NGP) fetch(g + G);
        const T* d = smem.e.dN + g * (NEN * 4);
        T A[9];
#pragma unroll
        for (int k = 0; k < 9; k++) A[k] = 0;
#pragma unroll
        for (int q = 0; q < NEN; q++) {
            T u0, u1, u2, d0, d1, d2;
            load3(su + (q * E + el) * 4, u0, u1, u2);
            load3(d + 4 * q, d0, d1, d2);
            A[0] += u0 * d0; A[1] += u0 * d1; A[2] += u0 * d2;
            A[3] += u1 * d0; A[4] += u1 * d1; A[5] += u1 * d2;
            A[6] += u2 * d0; A[7] += u2 * d1; A[8] += u2 * d2;
        }
        T H[9], P[9];
        const T* Jp = sJ + 9 * lane;
        {
            T Ji[9];
#pragma unroll
            for (int k = 0; k < 9; k++) Ji[k] = Jp[k];
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int j = 0; j < 3; j++)
                    H[3 * i + j] = A[3 * i] * Ji[j] + A[3 * i + 1] * Ji[3 + j] + A[3 * i + 2] * Ji[6 + j];
        }
        piola<T, MT>(*mp, H, P);
        const T wv = vol * __ldg(a.gw + g);
        T S[9];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const T j0 = Jp[3 * j], j1 = Jp[3 * j + 1], j2 = Jp[3 * j + 2];
#pragma unroll
            for (int i = 0; i < 3; i++) S[3 * i + j] = wv * (P[3 * i] * j0 + P[3 * i + 1] * j1 + P[3 * i + 2] * j2);
        }
#pragma unroll
        for (int q = 0; q < NEN; q++) {
            T d0, d1, d2;
            load3(d + 4 * q, d0, d1, d2);
#pragma unroll
            for (int i = 0; i < 3; i++) f[3 * q + i] += S[3 * i] * d0 + S[3 * i + 1] * d1 + S[3 * i + 2] * d2;
        }
        __syncwarp();
    }
    auto scatter = [&](int q, T f0, T f1, T f2) {
        const int node = __ldg(a.conn + static_cast<size_t>(q) * a.n + e);
        if (node >= a.n_free) return;
        if (a.contrib) {
            const size_t sl = a.slot0 + static_cast<size_t>(q) * a.n + e;
            a.contrib[sl] = static_cast<double>(f0);
            a.contrib[a.n_slots + sl] = static_cast<double>(f1);
            a.contrib[2 * a.n_slots + sl] = static_cast<double>(f2);
        } else {
            atomicAdd(a.r + 3 * node, static_cast<double>(f0));
            atomicAdd(a.r + 3 * node + 1, static_cast<double>(f1));
            atomicAdd(a.r + 3 * node + 2, static_cast<double>(f2));
        }
    };
    if constexpr (G == 1) {
        if (e < a.n) {
#pragma unroll
            for (int q = 0; q < NEN; q++) scatter(q, f[3 * q], f[3 * q + 1], f[3 * q + 2]);
        }
    } else {
        __syncthreads();  // u is no longer read
#pragma unroll
        for (int k = 0; k < 3 * NEN; k++) su[(part * 3 * NEN + k) * E + el] = f[k];
        __syncthreads();
        if (e < a.n)
            for (int q = part; q < NEN; q += G) {
                T s[3];
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    s[i] = su[(3 * q + i) * E + el];
#pragma unroll
                    for (int p = 1; p < G; p++) s[i] += su[(p * 3 * NEN + 3 * q + i) * E + el];
                }
                scatter(q, s[0], s[1], s[2]);
            }
    }
    griddep_launch();
}

// Deterministic scatter, second half: free node i adds its contributions in
// ascending slot order, r_i += sum_k contrib[gidx[k]], one thread per node
__global__ void __launch_bounds__(kBlock) k_gather(int n_free, const int* __restrict__ gptr,
    const int* __restrict__ gidx, const double* __restrict__ contrib, size_t n_slots, double* __restrict__ r)
{
    griddep_wait();
    const int i = blockIdx.x * kBlock + threadIdx.x;
    if (i >= n_free) return;
    double s0 = r[3 * i], s1 = r[3 * i + 1], s2 = r[3 * i + 2];
    for (int k = gptr[i]; k < gptr[i + 1]; k++) {
        const size_t sl = static_cast<size_t>(__ldg(gidx + k));
        s0 += __ldg(contrib + sl);
        s1 += __ldg(contrib + n_slots + sl);
        s2 += __ldg(contrib + 2 * n_slots + sl);
    }
    r[3 * i] = s0;
    r[3 * i + 1] = s1;
    r[3 * i + 2] = s2;
}

template <int NEN, int NGP, typename T, int BLK, bool Faces>
void launch_elem_law(const ElemArgs<T>& a, const FaceArgs<T>& fa, int ft, int mt, cudaStream_t st)
{
    constexpr int EPB = elems_per_cta<NGP, BLK>();
    const int grid = ft + (a.n + EPB - 1) / EPB;
    switch (mt) {
    case EFEM_NEO_HOOKEAN: launch_k(k_elem_residual<NEN, NGP, T, BLK, EFEM_NEO_HOOKEAN, Faces>, grid, BLK, 0, st, a, fa, ft); break;
    case EFEM_MOONEY_RIVLIN: launch_k(k_elem_residual<NEN, NGP, T, BLK, EFEM_MOONEY_RIVLIN, Faces>, grid, BLK, 0, st, a, fa, ft); break;
    case EFEM_YEOH: launch_k(k_elem_residual<NEN, NGP, T, BLK, EFEM_YEOH, Faces>, grid, BLK, 0, st, a, fa, ft); break;
    default: launch_k(k_elem_residual<NEN, NGP, T, BLK, -1, Faces>, grid, BLK, 0, st, a, fa, ft); break;
    }
}

template <int NEN, int NGP, typename T, int BLK>
void launch_elem_blk(const ElemArgs<T>& a, const FaceArgs<T>& fa, int mt, cudaStream_t st)
{
    constexpr int FPB = face_epb<NEN, BLK>();
    const int ft = (fa.n + FPB - 1) / FPB;
    if (ft > 0) launch_elem_law<NEN, NGP, T, BLK, true>(a, fa, ft, mt, st);
    else launch_elem_law<NEN, NGP, T, BLK, false>(a, fa, 0, mt, st);
}

template <int NEN, int NGP>
void launch_elem_thread(const ElemArgs<float>& a, const FaceArgs<float>& fa, int mt, cudaStream_t st, int per_sm)
{
    const size_t pad = per_sm < kPerSM ? kPadSmem : 0;
    constexpr int E = kTB / kSplit, FPB = face_epb<NEN, kTB>();
    const int ft = (fa.n + FPB - 1) / FPB, grid = ft + (a.n + E - 1) / E;
    switch (mt) {
    case EFEM_NEO_HOOKEAN: launch_k(k_elem_thread<NEN, NGP, EFEM_NEO_HOOKEAN, kSplit>, grid, kTB, pad, st, a, fa, ft); break;
    case EFEM_MOONEY_RIVLIN: launch_k(k_elem_thread<NEN, NGP, EFEM_MOONEY_RIVLIN, kSplit>, grid, kTB, pad, st, a, fa, ft); break;
    case EFEM_YEOH: launch_k(k_elem_thread<NEN, NGP, EFEM_YEOH, kSplit>, grid, kTB, pad, st, a, fa, ft); break;
    default: launch_k(k_elem_thread<NEN, NGP, -1, kSplit>, grid, kTB, pad, st, a, fa, ft); break;
    }
}

template <int NEN, int NGP, typename T>
void launch_elem(const DevBlock& b, const MatParams<T>* mats, const T* vol, const T* J0, const T* dN, const T* gw,
    int n_free, const double* u, double* r, cudaStream_t st, int threads, const Scatter& sc, const int* frozen,
    const FaceArgs<T>& fa, int per_sm)
{
    ElemArgs<T> a { b.n, n_free, b.conn, b.mat, vol, J0, dN, gw, mats, u, r, sc.contrib, sc.n_slots, sc.slot0,
        b.egroup, b.egroup ? frozen : nullptr };
    if constexpr (has_thread_kernel<T>(NEN, NGP))
        if (per_sm) return launch_elem_thread<NEN, NGP>(a, fa, b.mat_type, st, per_sm);
    if (threads == 64) launch_elem_blk<NEN, NGP, T, 64>(a, fa, b.mat_type, st);
    else if (threads == 256) launch_elem_blk<NEN, NGP, T, 256>(a, fa, b.mat_type, st);
    else launch_elem_blk<NEN, NGP, T, 128>(a, fa, b.mat_type, st);
}

// the element forces of block b and, with fa.n > 0, the pressure faces of its kind
template <typename T>
void dispatch_elem(const DevBlock& b, const MatParams<T>* mats, const T* vol, const T* J0, const T* dN, const T* gw,
    int n_free, const double* u, double* r, cudaStream_t st, int threads, const Scatter& sc = Scatter(),
    const int* frozen = nullptr, const FaceArgs<T>& fa = FaceArgs<T> {}, int per_sm = 0)
{
#define CASE(NEN, NGP)                                                                                 \
    if (b.nen == NEN && b.ngp == NGP) {                                                                \
        launch_elem<NEN, NGP, T>(b, mats, vol, J0, dN, gw, n_free, u, r, st, threads, sc, frozen, fa, per_sm); \
        return;                                                                                        \
    }
    CASE(4, 1)
    CASE(10, 4)
    CASE(10, 1)
    CASE(8, 8)
    CASE(8, 1)
    CASE(20, 27)
    CASE(20, 8)
#undef CASE
}

template <typename T>
FaceArgs<T> face_args(const DevFaces& f, const T* J0, const T* tw, const T* tN, const T* tdN, int n_free,
    const double* u, double* r, const Scatter& sc)
{
    const int gmax = *std::max_element(f.h_ngp.begin(), f.h_ngp.end());
    return FaceArgs<T> { f.n, n_free, gmax, f.conn, f.table, f.A0, J0, f.load, f.t_ngp, tw, tN, tdN, u, r, sc.contrib,
        sc.n_slots, sc.slot0 };
}

template <typename T>
void dispatch_face(int nen, const FaceArgs<T>& a, cudaStream_t st)
{
    auto grid_of = [&](int epb) { return (a.n + epb - 1) / epb; };
    switch (nen) {
    case 4: launch_k(k_face_residual<4, T>, grid_of(face_epb<4, kBlock>()), kBlock, 0, st, a); break;
    case 8: launch_k(k_face_residual<8, T>, grid_of(face_epb<8, kBlock>()), kBlock, 0, st, a); break;
    case 10: launch_k(k_face_residual<10, T>, grid_of(face_epb<10, kBlock>()), kBlock, 0, st, a); break;
    case 20: launch_k(k_face_residual<20, T>, grid_of(face_epb<20, kBlock>()), kBlock, 0, st, a); break;
    }
}

// The element block whose launch carries face set f: the first one with
// elements of the same kind (-1: none, all of that kind lack a material)
int block_of_faces(const Model& m, const DevFaces& f)
{
    for (size_t b = 0; b < m.blocks.size(); b++)
        if (m.blocks[b].n > 0 && m.blocks[b].nen == f.nen) return static_cast<int>(b);
    return -1;
}

// arguments of face set f, in the element kernels' precision
template <typename T>
FaceArgs<T> face_args_of(const Model& m, const DevFaces& f, const double* u, double* r, bool det)
{
    Scatter sc;
    if (det) sc = Scatter { m.d_contrib, m.n_slots, f.slot0 };
    if constexpr (sizeof(T) == 4)
        return face_args<float>(f, f.J0inv_f, f.t_w_f, f.t_N_f, f.t_dN_f, m.n_free, u, r, sc);
    else
        return face_args<double>(f, f.J0inv, f.t_w, f.t_N, f.t_dN, m.n_free, u, r, sc);
}

// the faces that go with element block bi (n = 0: none)
template <typename T>
FaceArgs<T> faces_with(const Model& m, size_t bi, const double* u, double* r, bool det)
{
    for (auto& f : m.faces)
        if (f.n > 0 && block_of_faces(m, f) == static_cast<int>(bi)) return face_args_of<T>(m, f, u, r, det);
    return FaceArgs<T> {};
}

}  // namespace

// Autotuner of the element kernels' CTA size: for every element block and
// both precisions, time the 64-, 128- and 256-thread variants and, where there
// is one, k_elem_thread with 8 and 7 CTAs per SM (2 warm-up and 5 timed launches each, with the faces
// that go along, CUDA events on the model's stream, at u = 0: the kernels' work
// does not depend on the values) and keep the fastest.
// opts.elem_threads = 64 / 128 / 256 forces one variant instead, and 1 forces
// k_elem_thread where there is one (the rest as with 0); so does
// deterministic mode (128 unless forced), so that every model and every solve
// runs the same instantiation and the results repeat bitwise whatever the
// timings.
int element_tune_key(const Model& m) { return m.opts.elem_threads | (m.opts.deterministic ? 0x400 : 0); }
efem_status tune_element_blocks(Model& m)
{
    const bool want_thread = m.opts.elem_threads == 1;
    const int forced = m.opts.elem_threads && !want_thread ? m.opts.elem_threads : (m.opts.deterministic ? 128 : 0);
    const size_t n = 3 * static_cast<size_t>(std::max(m.n_free, 1));
    EFEM_CUDA(cudaMemsetAsync(m.d_u, 0, n * sizeof(double), m.stream));
    cudaEvent_t e0, e1;
    EFEM_CUDA(cudaEventCreate(&e0));
    EFEM_CUDA(cudaEventCreate(&e1));
    for (size_t bi = 0; bi < m.blocks.size(); bi++) {
        DevBlock& b = m.blocks[bi];
        for (int prec = 0; prec < 2; prec++) {
            const bool has_thread = prec == 1 && has_thread_kernel<float>(b.nen, b.ngp);
            if (want_thread && has_thread) {
                b.threads[prec] = kTB;
                b.per_sm[prec] = kPerSM;
                continue;
            }
            if (forced == 64 || forced == 128 || forced == 256) {
                b.threads[prec] = forced;
                b.per_sm[prec] = 0;
                continue;
            }
            if (b.n == 0) {
                b.threads[prec] = 128;
                b.per_sm[prec] = 0;
                continue;
            }
            float best = 1e30f;
            for (int t : { 64, 128, 256, -kPerSM, 1 - kPerSM }) {  // negative: k_elem_thread, CTAs per SM
                if (t < 0 && !has_thread) continue;
                const int threads = t < 0 ? kTB : t, per_sm = t < 0 ? -t : 0;
                for (int rep = 0; rep < 7; rep++) {
                    if (rep == 2) EFEM_CUDA(cudaEventRecord(e0, m.stream));
                    if (prec == 1)
                        dispatch_elem<float>(b, m.d_mats_f, b.vol_f, b.J0inv_f, b.dN_f, b.gw_f, m.n_free, m.d_u, m.d_r,
                            m.stream, threads, Scatter(), nullptr, faces_with<float>(m, bi, m.d_u, m.d_r, false), per_sm);
                    else
                        dispatch_elem<double>(b, m.d_mats, b.vol, b.J0inv, b.dN, b.gw, m.n_free, m.d_u, m.d_r, m.stream,
                            threads, Scatter(), nullptr, faces_with<double>(m, bi, m.d_u, m.d_r, false), per_sm);
                }
                EFEM_CUDA(cudaEventRecord(e1, m.stream));
                EFEM_CUDA(cudaEventSynchronize(e1));
                float ms = 0.f;
                EFEM_CUDA(cudaEventElapsedTime(&ms, e0, e1));
                if (ms < best) {
                    best = ms;
                    b.threads[prec] = threads;
                    b.per_sm[prec] = per_sm;
                }
            }
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    EFEM_CUDA(cudaGetLastError());
    m.tuned_threads = element_tune_key(m);
    return EFEM_OK;
}

// kernels of one residual evaluation
int residual_launches(const Model& m)
{
    int n = 1 + (m.opts.deterministic ? 1 : 0);
    for (auto& b : m.blocks) n += b.n > 0;
    for (auto& f : m.faces) n += f.n > 0 && block_of_faces(m, f) < 0;
    return n;
}

efem_status launch_residual(Model& m, const double* d_u, double* d_r)
{
    return launch_residual_on(m, d_u, d_r, m.stream);
}

efem_status launch_residual_on(Model& m, const double* d_u, double* d_r, cudaStream_t stream,
    unsigned long long* stamp, bool init_r)
{
    const size_t n = 3 * static_cast<size_t>(m.n_free);
    if (n == 0) return EFEM_OK;
    // r = -f_ext (its first thread stores the start time in *stamp when given)
    extern void launch_neg(double* r, const double* f, size_t n, cudaStream_t st, unsigned long long* stamp);
    if (init_r) {
        launch_neg(d_r, m.d_fext, n, stream, stamp);
        m.launches++;
    }
    const bool mixed = m.opts.precision == EFEM_MIXED;
    const bool det = m.opts.deterministic != 0;
    if (det && !m.d_contrib) {
        set_error("deterministic scatter requested but its tables are not built");
        return EFEM_ERR_ARG;
    }
    for (size_t bi = 0; bi < m.blocks.size(); bi++) {
        const DevBlock& b = m.blocks[bi];
        if (b.n == 0) continue;
        m.launches++;
        Scatter sc;
        if (det) sc = Scatter { m.d_contrib, m.n_slots, b.slot0 };
        if (mixed)
            dispatch_elem<float>(b, m.d_mats_f, b.vol_f, b.J0inv_f, b.dN_f, b.gw_f, m.n_free, d_u, d_r, stream,
                b.threads[1], sc, m.d_frozen_groups, faces_with<float>(m, bi, d_u, d_r, det), b.per_sm[1]);
        else
            dispatch_elem<double>(b, m.d_mats, b.vol, b.J0inv, b.dN, b.gw, m.n_free, d_u, d_r, stream, b.threads[0], sc,
                m.d_frozen_groups, faces_with<double>(m, bi, d_u, d_r, det), b.per_sm[0]);
    }
    for (auto& f : m.faces) {
        if (f.n == 0 || block_of_faces(m, f) >= 0) continue;
        m.launches++;
        if (mixed)
            dispatch_face<float>(f.nen, face_args_of<float>(m, f, d_u, d_r, det), stream);
        else
            dispatch_face<double>(f.nen, face_args_of<double>(m, f, d_u, d_r, det), stream);
    }
    if (det) {
        launch_k(k_gather, (m.n_free + kBlock - 1) / kBlock, kBlock, 0, stream, m.n_free, m.d_gptr, m.d_gidx,
            m.d_contrib, m.n_slots, d_r);
        m.launches++;
    }
    EFEM_CUDA(cudaGetLastError());
    return EFEM_OK;
}

void free_gather(Model& m)
{
    dev_free(m.d_contrib);
    dev_free(m.d_gptr);
    dev_free(m.d_gidx);
    m.n_slots = 0;
}

// Slots of the deterministic scatter: element block b owns slots
// [slot0, slot0 + nen n) in node-major order, then each face group likewise;
// the gather lists of every free node are sorted by slot, so each node's sum
// has one fixed order whatever the launch configuration.
efem_status build_gather(Model& m)
{
    free_gather(m);
    size_t slots = 0;
    for (auto& b : m.blocks) {
        b.slot0 = slots;
        slots += static_cast<size_t>(b.nen) * b.n;
    }
    for (auto& f : m.faces) {
        f.slot0 = slots;
        slots += static_cast<size_t>(f.nen) * f.n;
    }
    if (slots >= static_cast<size_t>(INT_MAX)) {
        set_error("too many element-node pairs for the deterministic scatter");
        return EFEM_ERR_ARG;
    }
    std::vector<int> cnt(static_cast<size_t>(m.n_free) + 1, 0);
    auto node_of_slot = [&](auto&& visit) {
        for (auto& b : m.blocks)
            for (int a = 0; a < b.nen; a++)
                for (int e = 0; e < b.n; e++)
                    visit(b.h_conn[static_cast<size_t>(e) * b.nen + a], b.slot0 + static_cast<size_t>(a) * b.n + e);
        for (auto& f : m.faces)
            for (int q = 0; q < f.nen; q++)
                for (int k = 0; k < f.n; k++)
                    visit(f.h_conn[static_cast<size_t>(q) * f.n + k], f.slot0 + static_cast<size_t>(q) * f.n + k);
    };
    node_of_slot([&](int node, size_t) {
        if (node < m.n_free) cnt[node + 1]++;
    });
    for (int i = 0; i < m.n_free; i++) cnt[i + 1] += cnt[i];
    std::vector<int> idx(static_cast<size_t>(cnt[m.n_free]));
    std::vector<int> fill(cnt.begin(), cnt.end() - 1);
    node_of_slot([&](int node, size_t sl) {  // visited in ascending slot order
        if (node < m.n_free) idx[fill[node]++] = static_cast<int>(sl);
    });
    for (int i = 0; i < m.n_free; i++) std::sort(idx.begin() + cnt[i], idx.begin() + cnt[i + 1]);
    efem_status s;
    if ((s = dev_alloc(&m.d_contrib, 3 * std::max<size_t>(slots, 1))) != EFEM_OK) return s;
    if ((s = dev_upload(&m.d_gptr, cnt)) != EFEM_OK) return s;
    if (idx.empty()) idx.push_back(0);
    if ((s = dev_upload(&m.d_gidx, idx)) != EFEM_OK) return s;
    m.n_slots = slots;
    return EFEM_OK;
}

}  // namespace efem
