// Approximate-Jacobian Cholesky preconditioner on the GPU.
//
// Replaces the reference's Eigen SimplicialLLT factor of K~ = L (x) I3
// (src/simulation/nlsolver/LBFGS.h:65-81) and its solve inside the two-loop
// recursion (src/simulation/nlsolver/LBFGSMat.h:119-120).  The scalar node
// matrix L is factored (the same H0 = K~^{-1} up to rounding) and applied to
// the three displacement components at once.
//
// Numeric factorisation (multifrontal, one level of the supernodal
// elimination tree at a time, leaves first):
//   k_extend_add  one CTA per front: add the children's update blocks through
//                 the precomputed relative indices, children in a fixed order
//                 (the factor is bitwise repeatable);
//   k_diag, k_step  the inverse of the first 32 x 32 diagonal block's factor;
//                 then per 32-column step the panel, the update of the
//                 trailing triangle and the next block's inverse;
//   k_inverse     X = L_JJ^{-1} by doubling;
//   k_w           W = L_RJ X.  [X; W] is stored as one column-major matrix M
//                 per front, so the solves are matrix-vector products.
//
// Solve H0 v (3 right-hand sides interleaved per node): one persistent launch,
// k_solve below.  Every sum is formed in a fixed order (no atomics): results
// are deterministic.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>

#include "chol_symbolic.h"
#include "efem_internal.h"

namespace efem {

namespace {
constexpr int kFT = 256;  // factor threads
constexpr int kNB = 32;   // factor panel width
constexpr int kTS = 64;   // update tile
constexpr int kInvBatch = 8;  // steps between the inverse's launches
constexpr int kST = 256;  // solve threads

// one work item of the persistent triangular solve: a tile of a front, with
// all that a CTA has to know of the front, so that one load starts its work
struct alignas(16) SolveItem {
    int kind, s, r0, r1;    // front, rows (forward) or columns (backward) [r0, r1)
    int parent, r, c, f0;   // the front's parent, rows, columns, first column
    int nk, target, ptarget, pad;  // children; counts to wait for: own (children's updates, or own y), parent's x
    long long xw, rows, slot, upd; // offsets of M, of the row list, of the slot table, of the update vector
};

// a subtree solved by one CTA (see k_sub_fwd) and its chunks of factor rows
struct SubTree {
    int lo, hi;             // fronts [lo, hi] in postorder; hi is the root
    int j0, ncols;          // the subtree's columns [j0, j0 + ncols) (new numbering)
    int chunk0, nchunk_f;   // forward chunks
    int bchunk0, nchunk_b;  // backward chunks
};

struct SubChunk {
    int s;      // front
    int kind;   // 0: rows of L_JJ^{-1}; 1: rows of W; 2: rows of L_JJ^{-T} and of W^T
    int a, b;   // rows [a, b)
    int first;  // the front's first chunk of the sweep
};

constexpr int kSubStage = 4096;  // doubles per stage buffer (two buffers)
}  // namespace

struct Precond {
    Symbolic S;
    bool ready = false;     // symbolic analysis done and uploaded
    bool factored = false;  // numeric factor present
    bool ok = false;        // factor is positive definite
    double ms_factor = 0;
    int nlev = 0;
    // solve schedule: the persistent kernel's items, launch shape
    int n_items = 0, solve_grid = 1, solve_grid_full = 1, slots = 1;
    size_t solve_smem = 0;
    SolveItem* d_items = nullptr;
    std::vector<int> h_item_front;  // the front of every item (host)
    int* d_item_group = nullptr;    // batch unions: member of every item
    const int* d_frozen = nullptr;  // batch unions: per-member flag, 1 = skip its items
    int *d_parent = nullptr, *d_cnt = nullptr, *d_prow = nullptr;
    int* d_slot = nullptr;  // the fronts' slot tables (see SolveArgs)
    // subtree solves below the cut level (sub_levels levels of the tree)
    int sub_levels = 0, n_subs = 0;
    int sub_max_r = 0, sub_max_cols = 0, sub_max_depth = 0, sub_max_m = 0, sub_max_c = 0, sub_max_mroot = 0;
    size_t sub_smem_f = 0, sub_smem_b = 0;
    SubTree* d_subs = nullptr;
    SubChunk* d_chunks = nullptr;
    int *d_depth = nullptr, *d_xidx = nullptr;
    // factor schedule: per level the tiles of every 32-column step, and of the
    // products of the inverse's doublings (block size h) that follow step `after`
    struct Step {
        int k0, off, cnt;
    };
    struct Inv {
        int after, h, second, off, cnt;
    };
    std::vector<Step> steps;
    std::vector<Inv> invs;
    std::vector<int> lev_first_step, lev_first_inv;  // indices into steps and invs, nlev + 1
    int *d_first = nullptr, *d_ncol = nullptr, *d_nrow = nullptr, *d_child_ptr = nullptr,
        *d_child_list = nullptr, *d_relind = nullptr, *d_level_list = nullptr, *d_perm = nullptr, *d_fail = nullptr;
    long long *d_slot_off = nullptr, *d_front_off = nullptr, *d_rows_off = nullptr, *d_relind_off = nullptr, *d_xw_off = nullptr,
              *d_upd_off = nullptr, *d_a_pos = nullptr, *d_a_src = nullptr;
    int4* d_ea = nullptr;     // extend-add tiles (front, first row, first column)
    longlong2* d_zero = nullptr;  // spans of the fronts' own columns
    int n_zero = 0;
    std::vector<int> ea_off;  // nlev + 1
    double *d_xw = nullptr, *d_lp = nullptr;  // every front's M = [X; W], and its panels of L
    int4* d_wtiles = nullptr;  // (front, 64-row tile, 64-column tile) of every W
    std::vector<int> w_off;    // nlev + 1
    int4 *d_steps = nullptr, *d_invs = nullptr;  // tiles of k_step and k_inverse
    cudaStream_t capture2 = nullptr;  // second branch of the factorisation's graph
    int* d_res = nullptr;   // the last application's error flag
    int* h_flag = nullptr;  // mapped host memory: set by any application that gave up, cleared by the host
    double *d_front = nullptr, *d_upd = nullptr, *d_y = nullptr, *d_vals = nullptr;
    // graph replay of the numeric factorisation (the same launches every solve)
    cudaGraphExec_t factor_exec = nullptr;
    long long factor_launches = 0;
    cudaStream_t capture = nullptr;
};

namespace {

struct FrontArgs {
    const int *first, *ncol, *nrow, *child_ptr, *child_list, *relind;
    const int* slot;  // per front, child q, row t (slot_off[s] + q r + t): the update entry of that child landing on the row, or -1
    const long long *front_off, *rows_off, *relind_off, *xw_off, *upd_off, *slot_off;
    double* front;
    double* xw;  // per front M = [X; W], X = L_JJ^{-1} (c x c, zeros above the diagonal), W = L_RJ X ((r - c) x c):
                 // r x c column-major, leading dimension ld_of(r)
    double* lp;  // the panels L below the 32 x 32 diagonal blocks, laid out as M
    int* fail;
};

// leading dimension of a front's M: r rounded up to even, so that every
// column starts on a 16-byte boundary (the pad row holds zeros)
__host__ __device__ __forceinline__ long long ld_of(int r) { return (r + 1) & ~1; }


// ------------------------------------------------------------------ factorisation
__global__ void k_scatter_a(double* __restrict__ front, const long long* __restrict__ pos,
    const long long* __restrict__ src, const double* __restrict__ vals, long long n)
{
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
        front[pos[k]] = vals[src[k]];
}

// zeros in the fronts' own columns (the trailing parts are written before they
// are read); span = first double, count
__global__ void __launch_bounds__(kFT) k_zero(double* __restrict__ front, const longlong2* __restrict__ spans)
{
    const longlong2 sp = spans[blockIdx.x];
    for (long long i = threadIdx.x; i < sp.y; i += kFT) front[sp.x + i] = 0.0;
}

// Children's update blocks into the fronts of one level: one CTA per 64 rows x
// 32 columns of a front's lower triangle, every entry the sum over the
// children in order (no atomics: the factor is bitwise repeatable), read
// through the slot tables of the solve's assembly (entry of child q landing on
// row t, or -1).  Own columns hold L's entries and are added to; the trailing
// part is written, so nothing has to clear it.  Bound by memory once the
// chain slots -> children's entries is short: 12-47 us per level of the cap,
// with 165 MB cleared beforehand (own columns) instead of 836; one warp per
// column following the children's index lists took 32-48 us and needed all of
// the front cleared.
constexpr int kER = 64, kEC = 32;
__global__ void __launch_bounds__(kFT) k_extend_add(FrontArgs a, const int4* __restrict__ tiles)
{
    const int4 tl = tiles[blockIdx.x];
    const int s = tl.x, p0 = tl.y, q0 = tl.z;  // first row, first column
    const int r = a.nrow[s], c = a.ncol[s], k1 = a.child_ptr[s], k2 = a.child_ptr[s + 1];
    const int i = p0 + (threadIdx.x & (kER - 1)), jl = threadIdx.x >> 6;  // columns jl + 4 e
    double* F = a.front + a.front_off[s];
    griddep_wait();
    griddep_launch();
    double sum[kEC / 4];
#pragma unroll
    for (int e = 0; e < kEC / 4; e++) {
        const int j = q0 + jl + 4 * e;
        sum[e] = i < r && j < c && i >= j ? F[i + static_cast<long long>(j) * r] : 0.0;
    }
    for (int k = k1; k < k2; k++) {
        const int ch = a.child_list[k], rc = a.nrow[ch], cc = a.ncol[ch];
        const int* sl = a.slot + a.slot_off[s] + static_cast<long long>(k - k1) * r;
        const int b0 = static_cast<int>(a.upd_off[ch] / 3);
        const int si = i < r ? sl[i] : -1;
        const double* U = a.front + a.front_off[ch] + static_cast<long long>(cc) * rc + cc;
#pragma unroll
        for (int e = 0; e < kEC / 4; e++) {
            const int j = q0 + jl + 4 * e;
            const int sj = j <= i && j < r ? sl[j] : -1;
            if (si >= 0 && sj >= 0) sum[e] += U[static_cast<long long>(sj - b0) * rc + si - b0];
        }
    }
#pragma unroll
    for (int e = 0; e < kEC / 4; e++) {
        const int j = q0 + jl + 4 * e;
        if (i < r && j <= i) F[i + static_cast<long long>(j) * r] = sum[e];
    }
}

// ---- the 32-column steps of a level's fronts
//
// k_step, one launch per step k0: update tiles (ti, tj) form L = A X_kk^T on
// their two 64-row blocks of the step's columns -- a product with the inverse
// of the factored diagonal block, no substitution -- and subtract L_i L_j^T
// from their 64 x 64 tile of the trailing lower triangle.  The first tile of a
// row block keeps its L in the panel array; the front itself is only read in
// the step's columns, so no CTA can overtake another.  The tile that holds the
// next diagonal block then factors it and leaves its inverse for the next step
// (k_diag does so for the first), so the 32 pivots are done once per front and
// no launch waits for them alone.
//
// What bounds it: the chain of one step (load, product, update, 32 pivots of
// about 200 cycles) times the steps on the way to the root.  As three kernels,
// with a one-warp left-looking 32 x 32 Cholesky and one substitution per row, a
// step took 34 + 4 + 20 us (cold), now 13-20 us on the upper levels.  Whole
// factorisations: C3D8 beam 3.87 -> 1.37 ms, C3D20R cap 9.8 -> 3.85 ms, C3D10
// finger 10.4 -> 4.3 ms.  Every CTA repeating the block's elimination instead
// of taking the inverse from the step before: cap 4.6 ms; four pivots per
// exchange, for fewer barriers: slower (360 cycles per pivot).
constexpr int kStoreL = 1, kNextDiag = 2;        // tile.w
constexpr int kPS = kNB + 1, kXS = kNB + 2;      // shared-memory strides

__device__ __forceinline__ void cp8z(double* dst, const double* src, bool on)
{
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(on ? 8 : 0) : "memory");
}

// The inverse of the Cholesky factor of a kb x kb block (lower triangle in A:
// lane = row, columns w + 8 q of warp w; the identity past kb) into M.  The row
// operations that take the block to D^{1/2} L^T take the identity to L^{-1}, up
// to the rows' scaling.  The pivot column and the pivot row of X pass through
// shared memory; unrolled in full (200 cycles per pivot, 310 as a loop; one warp
// with the block in its registers needs 200 for the factor alone).
struct DiagSmem {
    double col[2][kNB], xrow[2][kNB];
};
__device__ __forceinline__ void diag_inverse(double (&A)[4], int kb, double* M, long long ld, int* fail, DiagSmem& sm)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double X[4], dl = 1.0;
    bool bad = false;
#pragma unroll
    for (int q = 0; q < 4; q++) X[q] = lane == w + 8 * q ? 1.0 : 0.0;
#pragma unroll
    for (int j = 0; j < kNB; j++) {
        const int jq = j >> 3, p = j & 1;
        if (w == (j & 7)) sm.col[p][lane] = A[jq];
        if (lane == j) {
#pragma unroll
            for (int q = 0; q <= jq; q++) sm.xrow[p][w + 8 * q] = X[q];
        }
        __syncthreads();
        double d = sm.col[p][j];
        if (!(d > 0.0)) {
            bad = true;
            d = 1.0;
        }
        const double f = lane > j ? sm.col[p][lane] * __drcp_rn(d) : 0.0;
        if (lane == j) dl = d;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (q >= jq) A[q] -= f * sm.col[p][w + 8 * q];
            if (q <= jq) X[q] -= f * sm.xrow[p][w + 8 * q];
        }
    }
    if (bad && threadIdx.x == 0) *fail = 1;
    const double sc = 1.0 / sqrt(dl);
#pragma unroll
    for (int q = 0; q < 4; q++)
        if (lane < kb && w + 8 * q < kb) M[(w + 8 * q) * ld + lane] = X[q] * sc;
}

// the first diagonal block of every front of a level
__global__ void __launch_bounds__(kFT) k_diag(FrontArgs a, const int* __restrict__ list)
{
    __shared__ DiagSmem sm;
    const int s = list[blockIdx.x], r = a.nrow[s], kb = min(kNB, a.ncol[s]);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double* F = a.front + a.front_off[s];
    double* M = a.xw + a.xw_off[s];
    griddep_wait();
    griddep_launch();
    double A[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int cc = w + 8 * q;
        A[q] = lane < kb && cc < kb ? (lane >= cc ? F[lane + static_cast<long long>(cc) * r] : 0.0) : (lane == cc ? 1.0 : 0.0);
    }
    diag_inverse(A, kb, M, ld_of(r), a.fail, sm);
}

// Rows [0, 64) of a panel (in P, row stride kPS) times X_kk^T: rows lane and
// lane + 32, columns 4 w + q (X_kk lower triangular: k <= 4 w + 3)
__device__ __forceinline__ void panel_times(const double* P, const double* XT, double (&o)[2][4])
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 4; q++) o[0][q] = o[1][q] = 0.0;
#pragma unroll 4
    for (int k = 0; k < 4 * w + 4; k++) {
        const double p0 = P[lane * kPS + k], p1 = P[(lane + 32) * kPS + k];
        const double2 xa = *reinterpret_cast<const double2*>(XT + k * kXS + 4 * w);
        const double2 xb = *reinterpret_cast<const double2*>(XT + k * kXS + 4 * w + 2);
        o[0][0] += p0 * xa.x;
        o[0][1] += p0 * xa.y;
        o[0][2] += p0 * xb.x;
        o[0][3] += p0 * xb.y;
        o[1][0] += p1 * xa.x;
        o[1][1] += p1 * xa.y;
        o[1][2] += p1 * xb.x;
        o[1][3] += p1 * xb.y;
    }
}

__global__ void __launch_bounds__(kFT, 3) k_step(FrontArgs a, const int4* __restrict__ tiles, int k0)
{
    __shared__ __align__(16) double XT[kNB * kXS];  // X_kk transposed: XT[k][j] = X_kk[j][k]
    __shared__ double buf[2 * kTS * kPS];           // panels Pi, Pj, then L of both
    __shared__ DiagSmem dsm;
    const int4 tl = tiles[blockIdx.x];
    const int s = tl.x;
    const int r = a.nrow[s], c = a.ncol[s], kb = min(kNB, c - k0), base = k0 + kb;
    // the trailing part of a front without children holds nothing before its first step
    const bool fresh = k0 == 0 && a.child_ptr[s] == a.child_ptr[s + 1];
    double* F = a.front + a.front_off[s];
    const long long mo = a.xw_off[s], ld = ld_of(r);
    double* M = a.xw + mo;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const bool two = tl.y != tl.z;  // off the diagonal: two row blocks
    const int i0 = base + tl.y * kTS, j0 = base + tl.z * kTS;
    double* Pi = buf;
    double* Pj = two ? buf + kTS * kPS : buf;
    griddep_wait();
    griddep_launch();
#pragma unroll
    for (int it = 0; it < kNB * kNB / kFT; it++) {
        const int idx = tid + it * kFT, j = idx & 31, k = idx >> 5;
        cp8z(XT + k * kXS + j, M + (k0 + min(k, kb - 1)) * ld + k0 + min(j, kb - 1), k < kb && j < kb);
    }
#pragma unroll
    for (int it = 0; it < kTS * kNB / kFT; it++) {
        const int idx = tid + it * kFT, p = idx & (kTS - 1), k = idx >> 6;
        const double* Fk = F + static_cast<long long>(k0 + min(k, kb - 1)) * r;
        cp8z(Pi + p * kPS + k, Fk + min(i0 + p, r - 1), k < kb && i0 + p < r);
        if (two) cp8z(Pj + p * kPS + k, Fk + min(j0 + p, r - 1), k < kb && j0 + p < r);
    }
    // tile rows (tid & 15) + 16 x, columns (tid >> 4) + 16 y
    const int ra = tid & 15, ca = tid >> 4;
    double acc[4][4];
#pragma unroll
    for (int y = 0; y < 4; y++)
#pragma unroll
        for (int x = 0; x < 4; x++) {
            const int gi = i0 + ra + 16 * x, gj = j0 + ca + 16 * y;
            acc[x][y] = gi < r && gi >= gj && !(fresh && gj >= c) ? F[gi + static_cast<long long>(gj) * r] : 0.0;
        }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    {
        double o[2][4], oj[2][4];
        panel_times(Pi, XT, o);
        if (two) panel_times(Pj, XT, oj);
        __syncthreads();
        double* Lp = a.lp + mo;
#pragma unroll
        for (int x = 0; x < 2; x++)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int row = lane + 32 * x, k = 4 * w + q;
                Pi[row * kPS + k] = o[x][q];
                if (two) Pj[row * kPS + k] = oj[x][q];
                if ((tl.w & kStoreL) && i0 + row < r && k < kb) Lp[(k0 + k) * ld + i0 + row] = o[x][q];
            }
    }
    __syncthreads();
#pragma unroll 2
    for (int k = 0; k < kb; k++) {
        double pa[4], pb[4];
#pragma unroll
        for (int x = 0; x < 4; x++) {
            pa[x] = Pi[(ra + 16 * x) * kPS + k];
            pb[x] = Pj[(ca + 16 * x) * kPS + k];
        }
#pragma unroll
        for (int x = 0; x < 4; x++)
#pragma unroll
            for (int y = 0; y < 4; y++) acc[x][y] -= pa[x] * pb[y];
    }
#pragma unroll
    for (int y = 0; y < 4; y++)
#pragma unroll
        for (int x = 0; x < 4; x++) {
            const int gi = i0 + ra + 16 * x, gj = j0 + ca + 16 * y;
            if (gi < r && gi >= gj) F[gi + static_cast<long long>(gj) * r] = acc[x][y];
        }
    if (!(tl.w & kNextDiag)) return;
    // the next step's diagonal block, rows and columns [0, 32) of this tile
    const int kn = min(kNB, c - base);
    __syncthreads();
#pragma unroll
    for (int y = 0; y < 2; y++)
#pragma unroll
        for (int x = 0; x < 2; x++) buf[(ra + 16 * x) * kPS + ca + 16 * y] = acc[x][y];
    __syncthreads();
    double A[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int cc = w + 8 * q;
        A[q] = lane < kn && cc < kn ? (lane >= cc ? buf[lane * kPS + cc] : 0.0) : (lane == cc ? 1.0 : 0.0);
    }
    diag_inverse(A, kn, M + base * ld + base, ld, a.fail, dsm);
}

// acc(64 x 64) += A(64 rows, k) B(k, 64 columns) over k in [k0, k1), 256
// threads, rows (tid & 15) + 16 x and columns (tid >> 4) + 16 y per thread
// (consecutive lanes on consecutive rows: no bank conflicts), in blocks of 16
// with the next block's operands fetched into registers while one is used.
// la(i, k) and lb(k, j) read an entry (0 outside).
constexpr int kGK = 16;
struct GemmSmem {
    double A[kGK][65], B[kGK][65];
};
template <typename LA, typename LB>
__device__ __forceinline__ void gemm64(GemmSmem& sm, double (&acc)[4][4], int k0, int k1, LA la, LB lb)
{
    const int tid = threadIdx.x, ti = tid & 15, tj = tid >> 4;
    double pa[4], pb[4];
    auto fetch = [&](int k) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int idx = tid + 256 * q;
            pa[q] = la(idx & 63, k + (idx >> 6));  // a warp on 32 consecutive rows of a column
            pb[q] = lb(k + (idx & 15), idx >> 4);  // 16 consecutive rows of two columns
        }
    };
    fetch(k0);
    for (int k = k0; k < k1; k += kGK) {
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int idx = tid + 256 * q;
            sm.A[idx >> 6][idx & 63] = pa[q];
            sm.B[idx & 15][idx >> 4] = pb[q];
        }
        __syncthreads();
        if (k + kGK < k1) fetch(k + kGK);
#pragma unroll 4
        for (int i = 0; i < kGK; i++) {
            double av[4], bv[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                av[q] = sm.A[i][ti + 16 * q];
                bv[q] = sm.B[i][tj + 16 * q];
            }
#pragma unroll
            for (int x = 0; x < 4; x++)
#pragma unroll
                for (int y = 0; y < 4; y++) acc[x][y] += av[x] * bv[y];
        }
    }
}

// X = L_JJ^{-1} from its 32 x 32 diagonal blocks, doubling the block size h:
// with X_11 and X_22 of two neighbouring blocks known,
//   X_21 = -X_22 (L_21 X_11),
// two products per doubling (second = 0: T = L_21 X_11 into the front's own
// columns, which nothing reads any more; second = 1: X_21).  Tiles: (front,
// first row of the pair, tile row * 64, tile column * 64).  log2(c / 32)
// doublings of dense products on a second branch of the graph, beside the
// steps of the levels above; one block row after another, as a chain of c / 32
// rows, took 0.76-0.87 ms.
__global__ void __launch_bounds__(256) k_inverse(FrontArgs a, const int4* __restrict__ tiles, int h, int second)
{
    __shared__ GemmSmem sm;
    const int4 tl = tiles[blockIdx.x];
    const int s = tl.x, p1 = tl.y, p2 = p1 + h, i0 = tl.z, j0 = tl.w;
    const int r = a.nrow[s], c = a.ncol[s], n2 = min(h, c - p2);  // rows of the second block
    const long long ld = ld_of(r);
    double* F = a.front + a.front_off[s];
    double* M = a.xw + a.xw_off[s];
    const double* Lp = a.lp + a.xw_off[s];
    double acc[4][4] = {};
    if (!second) {  // X_11 lower triangular: k >= column
        gemm64(sm, acc, j0 / kGK * kGK, h,
            [&](int i, int k) { return i0 + i < n2 && k < h ? Lp[(p1 + k) * ld + p2 + i0 + i] : 0.0; },
            [&](int k, int j) { return k < h && j0 + j < h ? M[(p1 + j0 + j) * ld + p1 + k] : 0.0; });
    } else {  // X_22 lower triangular: k <= row
        gemm64(sm, acc, 0, min(n2, i0 + 64),
            [&](int i, int k) { return i0 + i < n2 && k < n2 ? M[(p2 + k) * ld + p2 + i0 + i] : 0.0; },
            [&](int k, int j) { return k < n2 && j0 + j < h ? F[static_cast<long long>(p1 + j0 + j) * r + p2 + k] : 0.0; });
    }
    const int ti = threadIdx.x & 15, tj = threadIdx.x >> 4;
#pragma unroll
    for (int y = 0; y < 4; y++)
#pragma unroll
        for (int x = 0; x < 4; x++) {
            const int i = i0 + ti + 16 * x, j = j0 + tj + 16 * y;
            if (i >= n2 || j >= h) continue;
            if (second) M[(p1 + j) * ld + p2 + i] = -acc[x][y];
            else F[static_cast<long long>(p1 + j) * r + p2 + i] = acc[x][y];
        }
}

// W = L_RJ X for every front, one 64 x 64 tile of W per CTA, written into the
// rows below X in M.  With W the forward sweep forms a front's update
// g = f_R - W f_J without waiting for y_J, and the backward sweep forms
// x_J = L_JJ^{-T} y_J - W^T x_R in one step.
__global__ void __launch_bounds__(256) k_w(FrontArgs a, const int4* __restrict__ tiles)
{
    __shared__ GemmSmem sm;
    const int4 tl = tiles[blockIdx.x];
    const int s = tl.x, i0 = tl.y * 64, j0 = tl.z * 64;
    const int r = a.nrow[s], c = a.ncol[s], m = r - c;
    const long long ld = ld_of(r);
    double* M = a.xw + a.xw_off[s];
    const double* Lp = a.lp + a.xw_off[s];
    double acc[4][4] = {};
    gemm64(sm, acc, j0, c, [&](int i, int k) { return i0 + i < m && k < c ? Lp[k * ld + c + i0 + i] : 0.0; },
        [&](int k, int j) { return k < c && j0 + j < c ? M[(j0 + j) * ld + k] : 0.0; });
    const int ti = threadIdx.x & 15, tj = threadIdx.x >> 4;
#pragma unroll
    for (int y = 0; y < 4; y++)
#pragma unroll
        for (int x = 0; x < 4; x++) {
            const int i = i0 + ti + 16 * x, j = j0 + tj + 16 * y;
            if (i < m && j < c) M[j * ld + c + i] = acc[x][y];
        }
}

// ------------------------------------------------------------------ solves
//
// One persistent launch runs the whole solve H0 v (in place on v, 3 values per
// node).  Its work is a list of items in dependency order -- the forward
// sweep leaves first, then the backward sweep root first -- and every CTA
// takes the next item from a ticket counter.  An item waits until the items
// it depends on have finished (per-front completion counters), so a front
// starts as soon as its children (forward) or its parent (backward) are done,
// with no barrier between levels.  An item only waits on items with smaller
// tickets, which were taken by CTAs already running (a CTA takes its next
// ticket while it works on the current one, which keeps this true), so the
// wait always ends whatever the number of resident CTAs; each wait is still
// bounded, and a wait that runs out sets the error flag and makes every later
// wait give up.
//
// Both sweeps read the same matrix M = [X; W] of a front (X = L_JJ^{-1},
// W = L_RJ X, r x c column-major):
//   forward   M f_J:  y_J = X f_J and the update g = f_R - W f_J; f = b + the
//             children's updates
//   backward  x_J = M^T [y_J; -x_R]
// so an application reads nnz(L) doubles twice and holds them once: the
// backward sweep finds in L2 what the forward sweep read last, and a factor
// of up to about 100 MB stays there between applications.
//   * Forward tiles are rows of M.  A lane owns two consecutive rows (16-byte
//     loads; a warp reads up to 512 consecutive bytes of a column) and keeps
//     their sums in registers; what the rows leave of the CTA splits the
//     columns, and the partial sums meet in shared memory.
//   * Backward tiles are groups of four columns, one per warp (or several
//     warps splitting the rows of one): a lane takes two consecutive rows of
//     the four columns, so the vector in shared memory is read once for four
//     columns; one 12-value reduction over the lanes at the end.
//   * The vectors pass through shared memory in chunks of kVC entries, so the
//     kernel's shared memory does not depend on the fronts and every model
//     runs 3 CTAs per SM.
//   * All that can be had before the wait is fetched before it: the item's
//     record, the first kStage values of M of every thread (staged by the
//     thread that uses them, so no barrier stands between) and the rest of a
//     forward tile into L2, the index of every row to be assembled (a dense
//     table per front and child: consecutive threads read consecutive
//     entries), and the backward tile's part over y.
// What bounds it: on the beam and at the top of every tree the chain of
// dependent fronts (11-13 per sweep, 4-5 us each: notice 1, gather 0.8, product
// 1, partial sums and store 1, publish 0.5); on the cap and the finger below the
// top, where a level has about as many items as there are CTAs and the children
// are long done, the latencies of one item after another in its CTA (2 us from
// taking an item to being ready with nothing to wait for: record, indices,
// counter; gather 0.8-1, product 2-5, sums and publishing 2); not the bytes.  One application inside a solve, against four
// matrices staged through shared memory in 4-row tiles, and against M read
// into registers after the wait: C3D8 beam 124, 113, now 105 us; C3D20R cap
// 330, 192, now 182 us (281 MB, 1.5 TB/s); C3D10 finger 439, 241, now 226 us
// (340 MB, 1.5 TB/s).  More shared memory costs more than it gives (chunks of
// 1280 entries: cap 210 us; the index tables live in what L1 is left).
// Every sum has a fixed order (no atomics on data): results repeat bitwise.
enum ItemKind { kFwdTile = 0, kBwdTile = 1 };

constexpr int kVC = 896;       // vector entries (nodes) of a chunk in shared memory
constexpr int kMaxR = 256;     // most rows of a forward tile
constexpr int kFU = 4;         // columns a forward lane loads at a time beyond the staged ones
constexpr int kStage = 8;      // 16-byte values of M a thread stages before the wait
// doubles of M per tile (see precond_setup).  One application, beam / cap /
// finger, with kTileMin 1024, 2048, 4096: 115 / 192 / 242, 113 / 193 / 241,
// 119 / 192 / 238 us; with kTileMax 4096, 6144, 10240: 114 / 196 / 243,
// 113 / 193 / 241, 114 / 193 / 241 us.
constexpr int kTileMin = 2048, kTileMax = 6144;
constexpr int kRed = 8 * 64 * 3;  // doubles of the partial sums of a tile
constexpr size_t kSolveSmem = sizeof(double) * (3 * (kVC + kMaxR) + (kRed > 2 * kStage * kST ? kRed : 2 * kStage * kST));

// device counters, one int array: [cY ns][cGin ns][exits, ns - 1 unused][cX ns][ticket][error]
struct SolveArgs {
    FrontArgs a;
    const int* prow;          // per front row: the node's index in v
    const SolveItem* items;
    const int* slot;          // per front, child q, row t (item.slot + q r + t): the update entry of that child
                              // landing on the row, or -1
    int n_items, ns;
    double* v;
    double* y;
    double* upd;
    int* cnt;
    unsigned long long* stamp;  // when set: global timer at the start of the solve
    int spin_limit;             // polls of one wait before the solve gives up
    int test_wait;              // 1: the last item's wait target is raised by one (it can only run out)
    int n3;                     // entries of v (3 per free node)
    int *res, *hres;            // when set: this application's error flag, and a mapped host flag that stays set until the
                                // host clears it; the counters are left at zero
    const int* item_group;      // batch unions: the member each item belongs to
    const int* frozen;          // batch unions: 1 for a member that no longer iterates (its items are skipped)
};

constexpr int kSpinLimit = 1 << 22;  // default polls of one wait (about half a second)

__device__ __forceinline__ int ld_acquire(const int* p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// one thread: wait until *c >= target; false after `limit` polls (the
// error flag is then set) or when another wait has already given up.  The
// flag is read every 16th poll only: read every time, it doubled the time
// between two looks at the counter.
__device__ bool wait_ge(const int* c, int target, int* err, int limit)
{
    for (int it = 0;; it++) {
        if (ld_acquire(c) >= target) return true;
        if (it >= limit) {
            atomicExch(err, 1);
            return false;
        }
        if ((it & 15) == 15 && *reinterpret_cast<volatile int*>(err)) return false;
        __nanosleep(64);
    }
}

// count a finished tile: its results (made visible to this thread by the
// CTA's barrier) before the count
__device__ __forceinline__ void signal(int* c)
{
    asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(c) : "memory");
}

__device__ __forceinline__ void ld3(const double* p, double& a, double& b, double& c)
{
    a = __ldcg(p);
    b = __ldcg(p + 1);
    c = __ldcg(p + 2);
}

// The index of one row's assembly: the node of an own column (or -1) and the
// update entries of the first two children (or -1); loaded before the wait.
struct RowIdx {
    int v, g, h;
};
__device__ __forceinline__ RowIdx row_idx(const SolveArgs& A, const SolveItem& d, int t, bool valid)
{
    RowIdx x { -1, -1, -1 };
    if (!valid) return x;
    if (t < d.c) x.v = __ldg(A.prow + d.rows + t);
    if (d.nk > 0) x.g = __ldg(A.slot + d.slot + t);
    if (d.nk > 1) x.h = __ldg(A.slot + d.slot + d.r + t);
    return x;
}

// f on n1 front rows from t1 on and n2 rows from t2 on into dst (3 per row):
// the right-hand side on own columns (t < c) plus the children's update
// entries landing on the row, children in order.  The loads of two rows per
// thread (right-hand side and two children; more children follow) are issued
// before they are added; `ix` holds the first two rows' indices.
__device__ __forceinline__ void assemble(const SolveArgs& A, const SolveItem& d, int t1, int n1, int t2, int n2,
    double* dst, RowIdx (&ix)[2])
{
    const int n = n1 + n2;
    for (int i0 = threadIdx.x; i0 < n; i0 += 2 * kST) {
        double b[2][3], g[2][3], h[2][3];
#pragma unroll
        for (int u = 0; u < 2; u++) {
#pragma unroll
            for (int k = 0; k < 3; k++) b[u][k] = g[u][k] = h[u][k] = 0.0;
            if (ix[u].v >= 0) ld3(A.v + 3LL * ix[u].v, b[u][0], b[u][1], b[u][2]);
            if (ix[u].g >= 0) ld3(A.upd + 3LL * ix[u].g, g[u][0], g[u][1], g[u][2]);
            if (ix[u].h >= 0) ld3(A.upd + 3LL * ix[u].h, h[u][0], h[u][1], h[u][2]);
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {  // the next two rows' indices
            const int i = i0 + (u + 2) * kST;
            ix[u] = row_idx(A, d, i < n1 ? t1 + i : t2 + i - n1, i < n);
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int i = i0 + u * kST, t = i < n1 ? t1 + i : t2 + i - n1;
            if (i >= n) break;
#pragma unroll
            for (int k = 0; k < 3; k++) b[u][k] = b[u][k] + g[u][k] + h[u][k];
            for (int q = 2; q < d.nk; q++) {
                const int e = __ldg(A.slot + d.slot + static_cast<long long>(q) * d.r + t);
                if (e < 0) continue;
                double x0, x1, x2;
                ld3(A.upd + 3LL * e, x0, x1, x2);
                b[u][0] += x0;
                b[u][1] += x1;
                b[u][2] += x2;
            }
#pragma unroll
            for (int k = 0; k < 3; k++) dst[3 * i + k] = b[u][k];
        }
    }
}

// the indices of the first two rows per thread of a following assemble
__device__ __forceinline__ void first_idx(const SolveArgs& A, const SolveItem& d, int t1, int n1, int t2, int n2,
    RowIdx (&ix)[2])
{
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int i = threadIdx.x + u * kST;
        ix[u] = row_idx(A, d, i < n1 ? t1 + i : t2 + i - n1, i < n1 + n2);
    }
}

__device__ __forceinline__ void cp16(double2* dst, const double* src)
{
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ double2 ldm2(const double* p) { return __ldg(reinterpret_cast<const double2*>(p)); }

__device__ __forceinline__ void fma6(double* acc, double2 m, const double* f)
{
    const double f0 = f[0], f1 = f[1], f2 = f[2];
    acc[0] += m.x * f0;
    acc[1] += m.x * f1;
    acc[2] += m.x * f2;
    acc[3] += m.y * f0;
    acc[4] += m.y * f1;
    acc[5] += m.y * f2;
}

// two rows of four columns times z on these rows, added to the twelve sums
__device__ __forceinline__ void fma12(double (&acc)[4][3], const double2 (&m)[4], const double* z)
{
    const double2* zp = reinterpret_cast<const double2*>(z);
    const double2 za = zp[0], zc = zp[1], ze = zp[2];  // (z0 z1) (z2 z0') (z1' z2')
#pragma unroll
    for (int q = 0; q < 4; q++) {
        acc[q][0] += m[q].x * za.x;
        acc[q][1] += m[q].x * za.y;
        acc[q][2] += m[q].x * zc.x;
        acc[q][0] += m[q].y * zc.y;
        acc[q][1] += m[q].y * ze.x;
        acc[q][2] += m[q].y * ze.y;
    }
}

// twelve column sums (four columns x three components) over rows [i0, i1) of
// the chunk that starts at row zb (even), each lane two rows every `step`
__device__ __forceinline__ void cols_acc(double (&acc)[4][3], const double* const (&Mc)[4], const double* z, int zb,
    int i0, int i1, int step)
{
#pragma unroll 2
    for (int i = i0; i < i1; i += step) {
        double2 m[4];
#pragma unroll
        for (int q = 0; q < 4; q++) m[q] = ldm2(Mc[q] + i);
        fma12(acc, m, z + 3 * (i - zb));
    }
}

// the twelve sums over a warp: on return lane l holds the three components of
// column l >> 3 in acc[0]
__device__ __forceinline__ void cols_reduce(double (&acc)[4][3])
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < 2; q++)
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const double keep = lane & 16 ? acc[q + 2][k] : acc[q][k], send = lane & 16 ? acc[q][k] : acc[q + 2][k];
            acc[q][k] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
        }
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const double keep = lane & 8 ? acc[1][k] : acc[0][k], send = lane & 8 ? acc[0][k] : acc[1][k];
        double x = keep + __shfl_xor_sync(0xffffffffu, send, 8);
        x += __shfl_xor_sync(0xffffffffu, x, 4);
        x += __shfl_xor_sync(0xffffffffu, x, 2);
        x += __shfl_xor_sync(0xffffffffu, x, 1);
        acc[0][k] = x;
    }
}

__global__ void __launch_bounds__(kST, 3) k_solve(SolveArgs A)
{
    griddep_wait();
    extern __shared__ __align__(16) double sm[];
    double* vec = sm;                      // [kVC + kMaxR][3] chunk of the vector, and f on a tile's own below rows
    double* red = sm + 3 * (kVC + kMaxR);  // partial sums, once the staged values are used
    double2* stg = reinterpret_cast<double2*>(red) + threadIdx.x;  // the thread's staged values, kST apart
    __shared__ int item_sh, ok_sh, ok2_sh;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    int* ticket = A.cnt + 4 * A.ns;
    int* err = ticket + 1;
    if (tid == 0) {
        const int next = atomicAdd(ticket, 1);
        if (next == 0 && A.stamp) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            *A.stamp = t;
        }
        item_sh = next;
    }
    __syncthreads();
    for (;;) {
        const int it = item_sh;
        if (it >= A.n_items) {
            griddep_launch();  // no more items for this CTA
            break;
        }
        if (A.frozen && A.frozen[A.item_group[it]]) {
            // a batch member that stopped iterating: its tree of fronts (no
            // other member's items depend on it) is skipped whole
            __syncthreads();
            if (tid == 0) item_sh = atomicAdd(ticket, 1);
            __syncthreads();
            continue;
        }
        const int bump = A.test_wait && it == A.n_items - 1 ? 1 : 0;
        const SolveItem d = A.items[it];
        const long long ld = ld_of(d.r);
        const double* M = A.a.xw + d.xw;
        const int r0 = d.r0, r1 = d.r1, c = d.c;
        // The next ticket is drawn once this item's dependencies are in (a
        // few microseconds before the CTA is free), not when the item starts:
        // a CTA whose item waits on a long chain would otherwise hold up the
        // item of the ticket it drew.
        int next = 0;
        if (d.kind == kFwdTile) {
            // rows [r0, r1): 2^lsh row pairs per warp, 2^bsh blocks of 64 rows,
            // the rest of the CTA splits the columns
            const int R = r1 - r0, kend = min(c, r1);
            const int lsh = R <= 8 ? 2 : R <= 16 ? 3 : R <= 32 ? 4 : 5;
            const int bsh = R <= 64 ? 0 : R <= 128 ? 1 : 2;
            const int nw = 8 >> bsh, KS = nw << (5 - lsh);  // warps per block, column split
            const int lrow = ((w & ((1 << bsh) - 1)) << 6) + 2 * (lane & ((1 << lsh) - 1));
            const int wk = w >> bsh, ks = (wk << (5 - lsh)) + (lane >> lsh);
            const bool act = lrow < R;
            const double* Mr = M + r0 + lrow;
#pragma unroll
            for (int n = 0; n < kStage; n++)
                if (act && ks + n * KS < kend) cp16(stg + n * kST, Mr + (ks + n * KS) * ld);
            // the rest of a long row block at least into L2 (one lane per 64 bytes)
            if (act && (lane & 3) == 0)
                for (int q = ks + kStage * KS; q < kend; q += KS)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(Mr + q * ld));
            const int b0 = max(r0, c), nb = r1 - b0;  // the tile's below rows (nb <= 0: none)
            RowIdx ix[2];
            first_idx(A, d, 0, min(kend, kVC), b0, max(nb, 0), ix);
            if (tid == 0) {
                ok_sh = wait_ge(A.cnt + A.ns + d.s, d.target + bump, err, A.spin_limit);
                next = atomicAdd(ticket, 1);
            }
            __syncthreads();
            if (ok_sh) {
                double acc[6] = { 0, 0, 0, 0, 0, 0 };
                int k = ks;
                for (int kb = 0; kb < kend; kb += kVC) {
                    const int ke = min(kend, kb + kVC);
                    // own columns to vec; with the first chunk, the tile's below rows after them
                    if (kb > 0) {
                        __syncthreads();
                        first_idx(A, d, kb, ke - kb, 0, 0, ix);
                        assemble(A, d, kb, ke - kb, 0, 0, vec, ix);
                    } else {
                        assemble(A, d, 0, ke, b0, max(nb, 0), vec, ix);
                    }
                    __syncthreads();
                    if (act) {
                        if (kb == 0) {
                            stage_wait();  // a thread reads what it staged itself
#pragma unroll
                            for (int n = 0; n < kStage; n++)
                                if (ks + n * KS < ke) fma6(acc, stg[n * kST], vec + 3 * (ks + n * KS));
                            k = ks + kStage * KS;  // (a staged column lies in the first chunk: kStage KS <= 512)
                        }
                        while (k < ke) {
                            double2 buf[kFU];
#pragma unroll
                            for (int u = 0; u < kFU; u++)
                                buf[u] = k + u * KS < ke ? ldm2(Mr + (k + u * KS) * ld) : make_double2(0.0, 0.0);
#pragma unroll
                            for (int u = 0; u < kFU; u++)
                                if (k + u * KS < ke) fma6(acc, buf[u], vec + 3 * (k + u * KS - kb));
                            k += kFU * KS;
                        }
                        if (k >= ke) k = ke + ((ks - ke) % KS + KS) % KS;  // the first column of the next chunk
                    }
                }
                __syncthreads();  // the staged values make room for the partial sums
                for (int o = 1 << lsh; o < 32; o <<= 1)
#pragma unroll
                    for (int q = 0; q < 6; q++) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
                if (act && (lane >> lsh) == 0) {
                    double* o = red + (wk * (64 << bsh) + lrow) * 3;
#pragma unroll
                    for (int q = 0; q < 6; q++) o[q] = acc[q];
                }
                __syncthreads();
                const double* fr = vec + 3 * min(kend, kVC);
                for (int i = tid; i < 3 * R; i += kST) {
                    double x[8];
#pragma unroll
                    for (int h = 0; h < 8; h++) x[h] = h < nw ? red[h * (192 << bsh) + i] : 0.0;
                    const double sum = ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
                    if (i < 3 * (c - r0))
                        A.y[3LL * (d.f0 + r0) + i] = sum;
                    else
                        A.upd[d.upd + 3LL * (r0 - c) + i] = fr[i - 3 * (b0 - r0)] - sum;
                }
            }
            if (tid == 0) item_sh = next;
            __syncthreads();  // the item's results are written
            if (tid == 0) {
                if (r1 > c && d.parent >= 0) signal(A.cnt + A.ns + d.parent);
                if (r0 < c) signal(A.cnt + d.s);
            }
        } else {
            // columns [r0, r1), at most 32: one quad of columns per warp, or
            // (fewer than 8 quads) several warps splitting the quad's rows
            const int nq = (r1 - r0 + 3) >> 2;
            const int qsh = nq <= 1 ? 0 : nq <= 2 ? 1 : nq <= 4 ? 2 : 3;
            const int quad = w & ((1 << qsh) - 1), h = w >> qsh, wk = 8 >> qsh, step = 64 * wk;
            const bool act = quad < nq;
            const int* pr = A.prow + d.rows;
            const double* Mc[4];
#pragma unroll
            for (int q = 0; q < 4; q++) Mc[q] = M + min(r0 + 4 * quad + q, r1 - 1) * ld;
            // the first rows below the front's own, which are on the critical path
            const int zc = c & ~1, zi = zc + 64 * h + 2 * lane, zn = min(d.r, zc + kVC);
            if (act) {
#pragma unroll
                for (int n = 0; n < kStage / 4; n++)
                    if (zi + n * step < zn) {
#pragma unroll
                        for (int q = 0; q < 4; q++) cp16(stg + (4 * n + q) * kST, Mc[q] + zi + n * step);
                    }
            }
            if (tid == 0) {
                ok_sh = wait_ge(A.cnt + d.s, d.target + bump, err, A.spin_limit);
                if (!ok_sh) next = atomicAdd(ticket, 1);
            }
            __syncthreads();
            if (ok_sh) {
                double acc[4][3] = {};
                // own columns: y, this front's forward result
                for (int zb = r0 & ~1; zb < c; zb += kVC) {
                    const int ze = min(c, zb + kVC), zl = (ze + 1) & ~1, n = 3 * (ze - zb);
                    if (zb > r0) __syncthreads();
                    const double* y = A.y + 3LL * (d.f0 + zb);
#pragma unroll 4
                    for (int i = tid; i < 3 * (zl - zb); i += kST) vec[i] = i < n ? __ldcg(y + i) : 0.0;
                    __syncthreads();
                    if (act) cols_acc(acc, Mc, vec, zb, zb + 64 * h + 2 * lane, ze, step);
                }
                // below rows: -x of the ancestors, complete with the parent's
                int ip[4];
                const int io = tid < 3 * (r1 - r0) ? __ldg(pr + r0 + tid / 3) : 0;  // where the thread's result goes
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int t = zc + tid + u * kST;
                    ip[u] = t >= c && t < d.r ? __ldg(pr + t) : -1;
                }
                if (tid == 0) {
                    ok2_sh = d.parent < 0 || wait_ge(A.cnt + 3 * A.ns + d.parent, d.ptarget, err, A.spin_limit);
                    next = atomicAdd(ticket, 1);
                }
                __syncthreads();
                if (ok2_sh) {
                    for (int zb = zc; zb < d.r; zb += kVC) {
                        const int ze = min(d.r, zb + kVC), zl = (ze + 1) & ~1;
                        if (zb > zc) {
                            __syncthreads();
#pragma unroll
                            for (int u = 0; u < 4; u++) {
                                const int t = zb + tid + u * kST;
                                ip[u] = t < d.r ? __ldg(pr + t) : -1;
                            }
                        }
                        double x[4][3];
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            x[u][0] = x[u][1] = x[u][2] = 0.0;
                            if (ip[u] >= 0) ld3(A.v + 3LL * ip[u], x[u][0], x[u][1], x[u][2]);
                        }
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            const int i = tid + u * kST;
                            if (zb + i >= zl) break;
#pragma unroll
                            for (int k = 0; k < 3; k++) vec[3 * i + k] = -x[u][k];
                        }
                        __syncthreads();
                        int i = zb + 64 * h + 2 * lane;
                        if (act && zb == zc) {
                            stage_wait();
#pragma unroll
                            for (int n = 0; n < kStage / 4; n++, i += step)
                                if (i < ze) {
                                    const double2 m[4] = { stg[4 * n * kST], stg[(4 * n + 1) * kST], stg[(4 * n + 2) * kST],
                                        stg[(4 * n + 3) * kST] };
                                    fma12(acc, m, vec + 3 * (i - zb));
                                }
                        }
                        if (act) cols_acc(acc, Mc, vec, zb, i, ze, step);
                    }
                    __syncthreads();  // the staged values make room for the partial sums
                    cols_reduce(acc);
                    if ((lane & 7) == 0) {
                        double* o = red + ((h << qsh) + quad) * 12 + 3 * (lane >> 3);
#pragma unroll
                        for (int k = 0; k < 3; k++) o[k] = acc[0][k];
                    }
                    __syncthreads();
                    if (tid < 3 * (r1 - r0)) {
                        double x[8];
#pragma unroll
                        for (int q = 0; q < 8; q++) x[q] = q < wk ? red[(q << qsh) * 12 + tid] : 0.0;
                        A.v[3LL * io + tid % 3] = ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
                    }
                }
            }
            if (tid == 0) item_sh = next;
            __syncthreads();
            if (tid == 0) signal(A.cnt + 3 * A.ns + d.s);
        }
    }
    // The last CTA to leave.  A solve that gave up leaves v partly overwritten:
    // it is filled with NaN, so that a caller who cannot read the error flag (a
    // replayed graph) still sees that the result is not valid.  Then the flag
    // goes where it is read and the counters back to zero, so that no
    // application needs a launch to clear them.
    if (tid == 0) {
        __threadfence();
        ok_sh = atomicAdd(A.cnt + 2 * A.ns, 1) == static_cast<int>(gridDim.x) - 1;
        ok2_sh = *reinterpret_cast<volatile int*>(err);
    }
    __syncthreads();
    if (!ok_sh) return;
    __threadfence();
    if (ok2_sh)
        for (int i = tid; i < A.n3; i += kST) A.v[i] = __longlong_as_double(0x7ff8000000000000LL);
    if (A.res) {
        for (int i = tid; i < 4 * A.ns + 2; i += kST) A.cnt[i] = 0;
        if (tid == 0) {
            *A.res = ok2_sh;
            if (ok2_sh) *A.hres = 1;  // never cleared here: applications queued behind a failed one must not hide it
        }
    }
}

// ------------------------------------------------- staged row products (subtree solves)
__device__ __forceinline__ void cp8(double* dst, const double* src)
{
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
// rows [0, R) at src + row * ld, entries k in [max(lo0 + row, 0), L), into dst
// with row stride lp; one warp per row
__device__ __forceinline__ void stage_rows(double* dst, int lp, const double* src, long long ld, int R, int L, int lo0)
{
    const int lane = threadIdx.x & 31;
    for (int rr = threadIdx.x >> 5; rr < R; rr += kST / 32) {
        const double* sr = src + rr * ld;
        double* dr = dst + rr * lp;
        for (int k = max(lo0 + rr, 0) + lane; k < L; k += 32) cp8(dr + k, sr + k);
    }
}
// rows [0, R) of a column-major matrix (row q, column k at src[k ld + q]),
// entries k in [0, min(L, hi0 + row + 1)), into dst with row stride lp
__device__ __forceinline__ void stage_cols(double* dst, int lp, const double* src, long long ld, int R, int L, int hi0)
{
    for (int idx = threadIdx.x; idx < R * L; idx += kST) {
        const int k = idx / R, rr = idx - k * R;
        if (k < hi0 + rr + 1) cp8(dst + rr * lp + k, src + k * ld + rr);
    }
}
__device__ __forceinline__ void stage_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void stage_wait_but_one() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

__device__ __forceinline__ int odd(int L) { return L | 1; }
__device__ __forceinline__ int lanes_per_row(int R)
{
    int g = kST;
    while (g > 1 && (kST / g) < R) g >>= 1;
    return g;
}

// Dot products of staged rows [0, R) (row stride lp) with a 3-component vector
// v in shared memory (entry k at v[3 (k - vbase)]), over k in [lo, hi) with
// lo / hi for tri 0: 0 / L, 1: 0 / row0 + row + 1 (lower triangle), 2: row0 + row / L.  Each row gets a group of g threads (g = kST / R
// rounded to a power of two: a whole CTA for one row, one thread per row for
// kST rows); a group wider than a warp adds its warps' partial sums through
// shared memory.  Every sum has a fixed order.  out is called with
// (row, s0, s1, s2) by the first thread of each group.
template <typename Out>
__device__ __forceinline__ void rows_dot(const double* M, int lp, const double* v, int vbase, int R, int L, int tri,
    int row0, Out out)
{
    __shared__ double part[kST / 32][3];
    const int g = lanes_per_row(R);
    const int lig = threadIdx.x & (g - 1), grp = threadIdx.x / g, ngrp = kST / g;
    for (int base = 0; base < R; base += ngrp) {  // uniform trip count across the CTA
        const int rr = base + grp;
        const bool valid = rr < R;
        const int lo = !valid ? 0 : (tri == 2 ? row0 + rr : 0);
        const int hi = !valid ? 0 : (tri == 1 ? row0 + rr + 1 : L);
        const double* row = M + rr * lp;
        double a0 = 0, a1 = 0, a2 = 0, b0 = 0, b1 = 0, b2 = 0;
        int k = lo + lig;
        for (; k + g < hi; k += 2 * g) {
            const double d = row[k], e = row[k + g];
            const double* vv = v + 3 * (k - vbase);
            const double* vw = vv + 3 * g;
            a0 += d * vv[0];
            a1 += d * vv[1];
            a2 += d * vv[2];
            b0 += e * vw[0];
            b1 += e * vw[1];
            b2 += e * vw[2];
        }
        if (k < hi) {
            const double d = row[k];
            const double* vv = v + 3 * (k - vbase);
            a0 += d * vv[0];
            a1 += d * vv[1];
            a2 += d * vv[2];
        }
        a0 += b0;
        a1 += b1;
        a2 += b2;
        const int w = g < 32 ? g : 32;
        for (int o = w >> 1; o > 0; o >>= 1) {
            a0 += __shfl_xor_sync(0xffffffffu, a0, o);
            a1 += __shfl_xor_sync(0xffffffffu, a1, o);
            a2 += __shfl_xor_sync(0xffffffffu, a2, o);
        }
        if (g > 32) {  // several warps per row
            const int wid = threadIdx.x >> 5;
            if ((threadIdx.x & 31) == 0) {
                part[wid][0] = a0;
                part[wid][1] = a1;
                part[wid][2] = a2;
            }
            __syncthreads();
            if (valid && lig == 0) {
                a0 = a1 = a2 = 0.0;
                for (int q = wid; q < wid + g / 32; q++) {
                    a0 += part[q][0];
                    a1 += part[q][1];
                    a2 += part[q][2];
                }
                out(rr, a0, a1, a2);
            }
            __syncthreads();
        } else if (valid && lig == 0) {
            out(rr, a0, a1, a2);
        }
    }
}

// ---------------------------------------------------------------- subtree solves
// Below a cut level the elimination tree has many small fronts, and in the
// dataflow solve above every one of its levels costs an inter-CTA
// notification step (a few microseconds) per sweep.  There, each subtree is
// solved by one CTA from start to end instead: its fronts in postorder
// (forward) or reverse postorder (backward), the factor rows streamed through
// a double-buffered cp.async stage in chunks listed at set-up, and what passes
// between the subtree's fronts kept in shared memory -- the children's
// updates are added straight into the parent's assembly buffer (one buffer per
// depth below the subtree root), the solution on ancestor rows is read from
// the CTA's own copy.  Only the subtree root's update leaves the CTA (for its
// parent's assembly in k_solve), and the backward sweep reads the solution on
// the root's below rows once.  The subtree forward sweep runs before k_solve
// and the backward sweep after it, so the three launches need no counters.
// Sums keep the dataflow solve's order: b, then the children in list order.


struct SubArgs {
    FrontArgs a;
    const int* parent;
    const int* prow;
    const int* perm;
    const SubTree* subs;
    const SubChunk* chunks;
    const int* depth;  // per front: depth below its subtree root
    const int* xidx;   // per front row t >= c: >= 0 local column of the row; < 0: -(q + 1), the root's q-th below row
    int max_r, max_cols, max_depth, max_m, max_c, max_mroot;
    double* v;
    double* y;
    double* upd;
    unsigned long long* stamp;
};

__device__ __forceinline__ void sub_stage(const SubArgs& A, const SubChunk& ch, double* dst)
{
    const FrontArgs& a = A.a;
    const int s = ch.s, c = a.ncol[s], r = a.nrow[s], m = r - c, R = ch.b - ch.a;
    const int lc = odd(c), lm = odd(m);
    const double* M = a.xw + a.xw_off[s];
    const long long ld = ld_of(r);
    if (ch.kind == 0) {
        stage_cols(dst, lc, M + ch.a, ld, R, c, ch.a);
    } else if (ch.kind == 1) {
        stage_cols(dst, lc, M + c + ch.a, ld, R, c, c);
    } else {
        stage_rows(dst, lc, M + ch.a * ld, ld, R, c, ch.a);
        stage_rows(dst + R * lc, lm, M + ch.a * ld + c, ld, R, m, -R);
    }
    stage_commit();
}

// Forward sweep of one subtree per CTA: y_J = L_JJ^{-1} f_J for every front
// and the updates g = f_R - W f_J, added into the parent's buffer or, for the
// subtree root, written to the update array.
__global__ void __launch_bounds__(kST) k_sub_fwd(SubArgs A)
{
    extern __shared__ double sm[];
    double* buf[2] = { sm, sm + kSubStage };
    double* bsub = sm + 2 * kSubStage;          // [ncols][3] right-hand side on the subtree's columns
    double* acc = bsub + 3 * A.max_cols;        // [max_depth][max_r][3] assembly buffers
    const SubTree T = A.subs[blockIdx.x];
    const FrontArgs& a = A.a;
    if (A.stamp && blockIdx.x == 0 && threadIdx.x == 0) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        *A.stamp = t;
    }
    const int nch = T.nchunk_f;
    if (nch > 0) sub_stage(A, A.chunks[T.chunk0], buf[0]);
    for (int i = threadIdx.x; i < T.ncols; i += kST) {
        const double* src = A.v + 3LL * A.perm[T.j0 + i];
        bsub[3 * i] = src[0];
        bsub[3 * i + 1] = src[1];
        bsub[3 * i + 2] = src[2];
    }
    __syncthreads();
    for (int i = 0; i < nch; i++) {
        const SubChunk ch = A.chunks[T.chunk0 + i];
        if (i + 1 < nch) sub_stage(A, A.chunks[T.chunk0 + i + 1], buf[(i + 1) & 1]);
        const int s = ch.s, c = a.ncol[s], r = a.nrow[s], lc = odd(c);
        double* f = acc + static_cast<size_t>(A.depth[s]) * 3 * A.max_r;
        const bool inner = s != T.hi;  // the parent belongs to the subtree
        const int p = A.parent[s];
        if (ch.first) {
            if (a.child_ptr[s] == a.child_ptr[s + 1]) {  // no children: f = (b_J, 0)
                const int jc = a.first[s] - T.j0;
                for (int t = threadIdx.x; t < r; t += kST) {
                    const bool own = t < c;
                    f[3 * t] = own ? bsub[3 * (jc + t)] : 0.0;
                    f[3 * t + 1] = own ? bsub[3 * (jc + t) + 1] : 0.0;
                    f[3 * t + 2] = own ? bsub[3 * (jc + t) + 2] : 0.0;
                }
            }
            if (inner && a.child_list[a.child_ptr[p]] == s) {  // first child: open the parent's buffer
                double* fp = acc + static_cast<size_t>(A.depth[p]) * 3 * A.max_r;
                const int cp = a.ncol[p], rp = a.nrow[p], jp = a.first[p] - T.j0;
                for (int t = threadIdx.x; t < rp; t += kST) {
                    const bool own = t < cp;
                    fp[3 * t] = own ? bsub[3 * (jp + t)] : 0.0;
                    fp[3 * t + 1] = own ? bsub[3 * (jp + t) + 1] : 0.0;
                    fp[3 * t + 2] = own ? bsub[3 * (jp + t) + 2] : 0.0;
                }
            }
        }
        if (i + 1 < nch)
            stage_wait_but_one();
        else
            stage_wait();
        __syncthreads();
        const double* cur = buf[i & 1];
        const int R = ch.b - ch.a;
        if (ch.kind == 0) {
            double* yg = A.y + 3LL * (a.first[s] + ch.a);
            rows_dot(cur, lc, f, 0, R, c, 1, ch.a, [&](int rr, double y0, double y1, double y2) {
                yg[3 * rr] = y0;
                yg[3 * rr + 1] = y1;
                yg[3 * rr + 2] = y2;
            });
        } else {
            double* fp = inner ? acc + static_cast<size_t>(A.depth[p]) * 3 * A.max_r : nullptr;
            const int* rel = a.relind + a.relind_off[s];
            double* g = A.upd + a.upd_off[s];
            rows_dot(cur, lc, f, 0, R, c, 0, 0, [&](int rr, double d0, double d1, double d2) {
                const int q = ch.a + rr;
                const double* fq = f + 3 * (c + q);
                const double g0 = fq[0] - d0, g1 = fq[1] - d1, g2 = fq[2] - d2;
                if (inner) {
                    double* o = fp + 3 * rel[q];
                    o[0] += g0;
                    o[1] += g1;
                    o[2] += g2;
                } else {
                    g[3 * q] = g0;
                    g[3 * q + 1] = g1;
                    g[3 * q + 2] = g2;
                }
            });
        }
        __syncthreads();  // the buffer is free for the chunk after next; updates are visible
    }
}

// Backward sweep of one subtree per CTA, fronts root first:
// x_J = L_JJ^{-T} y_J - W^T x_R, x_R from the CTA's own copy of the solution.
__global__ void __launch_bounds__(kST) k_sub_bwd(SubArgs A)
{
    extern __shared__ double sm[];
    double* buf[2] = { sm, sm + kSubStage };
    double* ysub = sm + 2 * kSubStage;        // [ncols][3]
    double* xs = ysub + 3 * A.max_cols;       // [ncols][3] solution on the subtree's columns
    double* xr = xs + 3 * A.max_cols;         // [max_mroot][3] solution on the root's below rows
    double* xR = xr + 3 * A.max_mroot;        // [max_m][3] x_R of the current front
    double* tmp = xR + 3 * A.max_m;           // [max_c][3]
    const SubTree T = A.subs[blockIdx.x];
    const FrontArgs& a = A.a;
    const int nch = T.nchunk_b;
    if (nch > 0) sub_stage(A, A.chunks[T.bchunk0], buf[0]);
    for (int i = threadIdx.x; i < 3 * T.ncols; i += kST) ysub[i] = __ldcg(A.y + 3LL * T.j0 + i);
    {
        const int root = T.hi, cr = a.ncol[root], mr = a.nrow[root] - cr;
        const int* pr = A.prow + a.rows_off[root] + cr;
        for (int q = threadIdx.x; q < mr; q += kST) {
            const double* src = A.v + 3LL * pr[q];
            xr[3 * q] = __ldcg(src);
            xr[3 * q + 1] = __ldcg(src + 1);
            xr[3 * q + 2] = __ldcg(src + 2);
        }
    }
    __syncthreads();
    for (int i = 0; i < nch; i++) {
        const SubChunk ch = A.chunks[T.bchunk0 + i];
        if (i + 1 < nch) sub_stage(A, A.chunks[T.bchunk0 + i + 1], buf[(i + 1) & 1]);
        const int s = ch.s, c = a.ncol[s], m = a.nrow[s] - c, lc = odd(c), lm = odd(m);
        const long long ro = a.rows_off[s];
        const int jc = a.first[s] - T.j0;
        if (ch.first) {  // x on the front's below rows, from the subtree's columns or the root's below rows
            const int* xi = A.xidx + ro + c;
            for (int q = threadIdx.x; q < m; q += kST) {
                const int li = xi[q];
                const double* src = li >= 0 ? xs + 3 * li : xr + 3 * (-li - 1);
                xR[3 * q] = src[0];
                xR[3 * q + 1] = src[1];
                xR[3 * q + 2] = src[2];
            }
        }
        if (i + 1 < nch)
            stage_wait_but_one();
        else
            stage_wait();
        __syncthreads();
        const double* cur = buf[i & 1];
        const int R = ch.b - ch.a;
        rows_dot(cur, lc, ysub + 3 * jc, 0, R, c, 2, ch.a, [&](int rr, double x0, double x1, double x2) {
            tmp[3 * rr] = x0;
            tmp[3 * rr + 1] = x1;
            tmp[3 * rr + 2] = x2;
        });
        __syncthreads();
        const int* pr = A.prow + ro + ch.a;
        double* xo = xs + 3 * (jc + ch.a);
        rows_dot(cur + R * lc, lm, xR, 0, R, m, 0, 0, [&](int rr, double s0, double s1, double s2) {
            const double x0 = tmp[3 * rr] - s0, x1 = tmp[3 * rr + 1] - s1, x2 = tmp[3 * rr + 2] - s2;
            xo[3 * rr] = x0;
            xo[3 * rr + 1] = x1;
            xo[3 * rr + 2] = x2;
            double* o = A.v + 3LL * pr[rr];
            o[0] = x0;
            o[1] = x1;
            o[2] = x2;
        });
        __syncthreads();
    }
}

FrontArgs args_of(Precond& P)
{
    return FrontArgs { P.d_first, P.d_ncol, P.d_nrow, P.d_child_ptr, P.d_child_list, P.d_relind, P.d_slot, P.d_front_off,
        P.d_rows_off, P.d_relind_off, P.d_xw_off, P.d_upd_off, P.d_slot_off, P.d_front, P.d_xw, P.d_lp, P.d_fail };
}

// the work buffers of one solve
struct SolveBufs {
    double* y;    // forward result, 3 per node
    double* upd;  // fronts' update vectors
    int* cnt;     // completion counters, ticket, error flag (4 ns + 2)
};

// limits of the persistent solve's device-side waits (efem_options.wait_limit, wait_test)
struct WaitCfg {
    int limit, test;
};
WaitCfg wait_cfg(const Model& m)
{
    return WaitCfg { m.opts.wait_limit > 0 ? m.opts.wait_limit : kSpinLimit, m.opts.wait_test ? 1 : 0 };
}

// Enqueue one H0 application on stream st.  With the model's own work buffers
// (own) the counters are zero beforehand and left so; other buffers' are
// cleared first and keep the error flag.
efem_status enqueue_solve(const Precond& P, const FrontArgs& a, const SolveBufs& b, double* d_v, cudaStream_t st,
    WaitCfg wc, bool own, unsigned long long* stamp = nullptr)
{
    const int ns = P.S.ns;
    if (!own) EFEM_CUDA(cudaMemsetAsync(b.cnt, 0, sizeof(int) * (4 * static_cast<size_t>(ns) + 2), st));
    const SubArgs B { a, P.d_parent, P.d_prow, P.d_perm, P.d_subs, P.d_chunks, P.d_depth, P.d_xidx, P.sub_max_r,
        P.sub_max_cols, P.sub_max_depth, P.sub_max_m, P.sub_max_c, P.sub_max_mroot, d_v, b.y, b.upd, stamp };
    if (P.n_subs > 0) k_sub_fwd<<<P.n_subs, kST, P.sub_smem_f, st>>>(B);
    SolveArgs A { a, P.d_prow, P.d_items, P.d_slot, P.n_items, ns, d_v, b.y, b.upd, b.cnt,
        P.n_subs > 0 ? nullptr : stamp, wc.limit, wc.test, 3 * P.S.n, own ? P.d_res : nullptr, own ? P.h_flag : nullptr,
        P.d_item_group, P.d_item_group ? P.d_frozen : nullptr };
    if (P.n_items > 0) launch_k(k_solve, P.solve_grid, kST, P.solve_smem, st, A);
    if (P.n_subs > 0) k_sub_bwd<<<P.n_subs, kST, P.sub_smem_b, st>>>(B);
    return EFEM_OK;
}

}  // namespace

void free_precond(Model& m)
{
    if (!m.precond) return;
    m.epoch++;
    Precond& P = *m.precond;
    if (P.factor_exec) cudaGraphExecDestroy(P.factor_exec);
    if (P.capture) cudaStreamDestroy(P.capture);
    if (P.capture2) cudaStreamDestroy(P.capture2);
    if (P.h_flag) cudaFreeHost(P.h_flag);
    for (int** p : { &P.d_first, &P.d_ncol, &P.d_nrow, &P.d_child_ptr, &P.d_child_list, &P.d_relind,
             &P.d_level_list, &P.d_perm, &P.d_fail, &P.d_parent, &P.d_cnt, &P.d_res, &P.d_prow, &P.d_depth, &P.d_xidx, &P.d_slot })
        dev_free(*p);
    for (long long** p : { &P.d_slot_off, &P.d_front_off, &P.d_rows_off, &P.d_relind_off, &P.d_xw_off, &P.d_upd_off, &P.d_a_pos,
             &P.d_a_src })
        dev_free(*p);
    dev_free(P.d_ea);
    dev_free(P.d_zero);
    dev_free(P.d_items);
    dev_free(P.d_item_group);
    dev_free(P.d_subs);
    dev_free(P.d_chunks);
    dev_free(P.d_steps);
    dev_free(P.d_invs);
    dev_free(P.d_wtiles);
    for (double** p : { &P.d_front, &P.d_xw, &P.d_lp, &P.d_upd, &P.d_y, &P.d_vals })
        dev_free(*p);
    delete m.precond;
    m.precond = nullptr;
}

void precond_info(const Model& m, efem_model_info* info)
{
    if (!m.precond) return;
    const Symbolic& S = m.precond->S;
    info->factor_nnz = S.nnz_L;
    info->n_supernodes = S.ns;
    info->n_levels = static_cast<int>(S.level_ptr.size()) - 1;
    info->factor_gflop = S.flops * 1e-9;
    long long dn = 0;
    for (int s = 0; s < S.ns; s++) dn += static_cast<long long>(S.ncol[s]) * (S.ncol[s] + 1) / 2;
    info->factor_dinv_nnz = dn;
    info->solve_subtree_levels = m.precond->sub_levels;
    info->n_solve_subtrees = m.precond->n_subs;
    info->solve_ctas = m.precond->solve_grid;
    info->solve_smem_bytes = static_cast<int>(m.precond->solve_smem);
}

thread_local int t_batch = 0;

// the persistent solve's grid for the calling thread (see precond_sync_grid)
static int solve_grid_for(const Precond& P)
{
    if (t_batch <= 0) return P.solve_grid_full;
    return std::max(1, std::min(P.n_items, P.slots / t_batch));
}

static efem_status precond_factor(Model& m, int* ok, double* ms_factor);

efem_status precond_setup(Model& m, bool refactor, int* ok, double* ms_factor)
{
    if (m.precond && m.precond->factored && !refactor) {
        *ok = m.precond->ok;
        *ms_factor = 0.0;
        return EFEM_OK;
    }
    if (m.precond && m.precond->ready) return precond_factor(m, ok, ms_factor);
    free_precond(m);
    m.precond = new Precond();
    Precond& P = *m.precond;
    Symbolic& S = P.S;
    // host: assemble L, order, analyse
    std::vector<int> rp, ci;
    std::vector<double> vals;
    assemble_L_csr(m, rp, ci, vals);
    std::vector<double> coords(3 * static_cast<size_t>(m.n_free));
    for (int i = 0; i < m.n_free; i++)
        for (int k = 0; k < 3; k++) coords[3 * i + k] = m.X[3 * static_cast<size_t>(m.node_of_dnode[i]) + k];
    symbolic_analysis(m.n_free, rp, ci, coords.data(), S);
    P.nlev = static_cast<int>(S.level_ptr.size()) - 1;
    const int nlev = P.nlev;
    // solve and factor schedules
    std::vector<int4> ea;
    std::vector<longlong2> zeros;
    for (int s = 0; s < S.ns; s++) {
        const long long n = static_cast<long long>(S.nrow[s]) * S.ncol[s], step = 16384;
        for (long long o = 0; o < n; o += step) zeros.push_back(make_longlong2(S.front_off[s] + o, std::min(step, n - o)));
    }
    P.n_zero = static_cast<int>(zeros.size());
    P.ea_off.assign(1, 0);
    P.w_off.assign(1, 0);
    std::vector<int4> steps, invs, wtiles;
    P.lev_first_step.assign(1, 0);
    P.lev_first_inv.assign(1, 0);
    for (int l = 0; l < nlev; l++) {
        int maxc = 0;
        for (int q = S.level_ptr[l]; q < S.level_ptr[l + 1]; q++) {
            const int s = S.level_list[q];
            const int c = S.ncol[s], mm = S.nrow[s] - c;
            maxc = std::max(maxc, c);
            if (S.child_ptr[s + 1] > S.child_ptr[s])
                for (int j = 0; j < S.nrow[s]; j += kEC)
                    for (int i = j / kER * kER; i < S.nrow[s]; i += kER) ea.push_back(make_int4(s, i, j, 0));
            for (int tk = 0; tk * 64 < mm; tk++)
                for (int tj = 0; tj * 64 < c; tj++) wtiles.push_back(make_int4(s, tk, tj, 0));
        }
        P.ea_off.push_back(static_cast<int>(ea.size()));
        P.w_off.push_back(static_cast<int>(wtiles.size()));
        for (int k0 = 0; k0 < maxc; k0 += kNB) {
            Precond::Step st { k0, static_cast<int>(steps.size()), 0 };
            for (int q = S.level_ptr[l]; q < S.level_ptr[l + 1]; q++) {
                const int s = S.level_list[q];
                const int c = S.ncol[s], r = S.nrow[s];
                if (c <= k0) continue;
                const int nt = (r - k0 - std::min(kNB, c - k0) + kTS - 1) / kTS;
                for (int tj = 0; tj < nt; tj++)
                    for (int ti = tj; ti < nt; ti++)
                        steps.push_back(make_int4(s, ti, tj, (tj == 0 ? kStoreL : 0) | (ti == 0 && c > k0 + kNB ? kNextDiag : 0)));
            }
            st.cnt = static_cast<int>(steps.size()) - st.off;
            P.steps.push_back(st);
        }
        P.lev_first_step.push_back(static_cast<int>(P.steps.size()));
        // Doublings of the inverse, as soon as their blocks are there: the first
        // product (L_21 X_11) after X_11's last step, the second after X_22's,
        // in batches of kInvBatch steps.  Within a batch sizes ascend.
        const int nsteps = (maxc + kNB - 1) / kNB;
        for (int batch = 0; batch < nsteps; batch += kInvBatch) {
            const int last = std::min(nsteps, batch + kInvBatch) - 1;  // step after which the batch runs
            for (int h = kNB; h < maxc; h *= 2)
                for (int second = 0; second < 2; second++) {
                    Precond::Inv st { last, h, second, static_cast<int>(invs.size()), 0 };
                    for (int q = S.level_ptr[l]; q < S.level_ptr[l + 1]; q++) {
                        const int s = S.level_list[q], c = S.ncol[s];
                        for (int p1 = 0; p1 + h < c; p1 += 2 * h) {
                            const int ready = ((second ? std::min(c, p1 + 2 * h) : p1 + h) + kNB - 1) / kNB - 1;
                            if (ready < batch || ready > last) continue;
                            for (int i = 0; i < std::min(h, c - p1 - h); i += 64)
                                for (int j = 0; j < h; j += 64) invs.push_back(make_int4(s, p1, i, j));
                        }
                    }
                    st.cnt = static_cast<int>(invs.size()) - st.off;
                    if (st.cnt > 0) P.invs.push_back(st);
                }
        }
        P.lev_first_inv.push_back(static_cast<int>(P.invs.size()));
    }
    auto odd_h = [](int L) { return L | 1; };
    // Subtree solves: fronts on the lowest K levels are solved per subtree by
    // one CTA (k_sub_fwd / k_sub_bwd), the levels above by the dataflow
    // k_solve.  opts.solve_subtree_levels = K asks for them (K is lowered
    // until the subtrees fit in shared memory); the default (-1) is K = 0.
    // Measured on the 20 480-element C3D8 beam (11 levels), one H0
    // application inside the solve costs 106 us with K = 0 and 125, 152, 186,
    // 283 us with K = 1, 2, 3, 4: a subtree CTA streams its
    // factor rows one 32 KB chunk ahead, about 20 GB/s, and works through its
    // fronts one after another, which is slower than the notification steps
    // of the levels it replaces.
    std::vector<int> lev(S.ns, 0), nsub(S.ns, 1), sdepth(S.ns, 0);
    for (int l = 0; l < nlev; l++)
        for (int q = S.level_ptr[l]; q < S.level_ptr[l + 1]; q++) lev[S.level_list[q]] = l;
    for (int s = 0; s < S.ns; s++)
        if (S.parent[s] >= 0) nsub[S.parent[s]] += nsub[s];
    bool postorder = true;  // every subtree is the index range [s - nsub[s] + 1, s]
    for (int s = 0; s < S.ns && postorder; s++)
        for (int k = s - nsub[s] + 1; k < s && postorder; k++) {
            int u = k;
            while (u >= 0 && u < s) u = S.parent[u];
            postorder = u == s;
        }
    struct SubPlan {
        bool ok = true;
        int max_r = 1, max_cols = 1, max_depth = 1, max_m = 1, max_c = 1, max_mroot = 1;
        size_t smem_f = 0, smem_b = 0;
        std::vector<int> roots;
    };
    auto plan = [&](int K) {
        SubPlan p;
        if (K <= 0) return p;
        for (int s = 0; s < S.ns; s++)
            if (lev[s] < K && (S.parent[s] < 0 || lev[S.parent[s]] >= K)) p.roots.push_back(s);
        for (int root : p.roots) {
            int cols = 0;
            for (int k = root; k > root - nsub[root]; k--) {  // parents before children
                sdepth[k] = k == root ? 0 : sdepth[S.parent[k]] + 1;
                const int c = S.ncol[k], r = S.nrow[k], mm = r - c;
                cols += c;
                p.max_r = std::max(p.max_r, r);
                p.max_m = std::max(p.max_m, mm);
                p.max_c = std::max(p.max_c, c);
                p.max_depth = std::max(p.max_depth, sdepth[k] + 1);
                if (odd_h(c) + odd_h(mm) > kSubStage) p.ok = false;
            }
            p.max_cols = std::max(p.max_cols, cols);
            p.max_mroot = std::max(p.max_mroot, S.nrow[root] - S.ncol[root]);
        }
        p.smem_f = sizeof(double) * (2 * static_cast<size_t>(kSubStage) + 3 * static_cast<size_t>(p.max_cols)
            + 3 * static_cast<size_t>(p.max_depth) * p.max_r);
        p.smem_b = sizeof(double) * (2 * static_cast<size_t>(kSubStage) + 6 * static_cast<size_t>(p.max_cols)
            + 3 * static_cast<size_t>(p.max_mroot + p.max_m + p.max_c));
        if (std::max(p.smem_f, p.smem_b) > 200 * 1024) p.ok = false;
        return p;
    };
    int K = 0;
    if (postorder && m.opts.solve_subtree_levels > 0)
        for (K = std::min(m.opts.solve_subtree_levels, nlev); K > 0 && !plan(K).ok; K--) {
        }
    const SubPlan sp = plan(K);  // also leaves sdepth for the chosen subtrees
    std::vector<char> in_sub(S.ns, 0);
    for (int s = 0; s < S.ns; s++) in_sub[s] = lev[s] < K;
    std::vector<SubTree> subs;
    std::vector<SubChunk> chunks;
    std::vector<int> xidx(S.rows.size(), 0);
    for (int root : sp.roots) {
        SubTree T {};
        T.lo = root - nsub[root] + 1;
        T.hi = root;
        T.j0 = S.first[T.lo];
        T.ncols = S.first[root] + S.ncol[root] - T.j0;
        T.chunk0 = static_cast<int>(chunks.size());
        for (int k = T.lo; k <= T.hi; k++) {
            const int c = S.ncol[k], mm = S.nrow[k] - c, rx = std::max(1, kSubStage / odd_h(c));
            for (int a0 = 0; a0 < c; a0 += rx) chunks.push_back(SubChunk { k, 0, a0, std::min(c, a0 + rx), a0 == 0 });
            for (int a0 = 0; a0 < mm; a0 += rx) chunks.push_back(SubChunk { k, 1, a0, std::min(mm, a0 + rx), 0 });
        }
        T.nchunk_f = static_cast<int>(chunks.size()) - T.chunk0;
        T.bchunk0 = static_cast<int>(chunks.size());
        for (int k = T.hi; k >= T.lo; k--) {
            const int c = S.ncol[k], mm = S.nrow[k] - c, rb = std::max(1, kSubStage / (odd_h(c) + odd_h(mm)));
            for (int a0 = 0; a0 < c; a0 += rb) chunks.push_back(SubChunk { k, 2, a0, std::min(c, a0 + rb), a0 == 0 });
            // below rows: a column of the subtree, or one of the root's below rows
            const long long ro = S.rows_off[k];
            const int* rb0 = S.rows.data() + S.rows_off[root] + S.ncol[root];
            const int nrb = S.nrow[root] - S.ncol[root];
            for (int t = c; t < S.nrow[k]; t++) {
                const int row = S.rows[ro + t];
                if (row >= T.j0 && row < T.j0 + T.ncols) {
                    xidx[ro + t] = row - T.j0;
                } else {
                    const int q = static_cast<int>(std::lower_bound(rb0, rb0 + nrb, row) - rb0);
                    if (q >= nrb || rb0[q] != row) {
                        set_error("internal: a subtree row is neither a subtree column nor a root row");
                        return EFEM_ERR_CUDA;
                    }
                    xidx[ro + t] = -(q + 1);
                }
            }
        }
        T.nchunk_b = static_cast<int>(chunks.size()) - T.bchunk0;
        subs.push_back(T);
    }
    P.sub_levels = K;
    P.n_subs = static_cast<int>(subs.size());
    P.sub_max_r = sp.max_r;
    P.sub_max_cols = sp.max_cols;
    P.sub_max_depth = sp.max_depth;
    P.sub_max_m = sp.max_m;
    P.sub_max_c = sp.max_c;
    P.sub_max_mroot = sp.max_mroot;
    P.sub_smem_f = sp.smem_f;
    P.sub_smem_b = sp.smem_b;
    // Storage of the fronts' M = [X; W] and the slot tables of the assembly.
    std::vector<long long> xw_off(S.ns + 1, 0), slot_off(S.ns + 1, 0);
    for (int s = 0; s < S.ns; s++) {
        xw_off[s + 1] = xw_off[s] + ld_of(S.nrow[s]) * S.ncol[s];
        slot_off[s + 1] = slot_off[s] + static_cast<long long>(S.child_ptr[s + 1] - S.child_ptr[s]) * S.nrow[s];
    }
    const long long xw_size = xw_off[S.ns];
    std::vector<int> slot(static_cast<size_t>(slot_off[S.ns]), -1);
    for (int s = 0; s < S.ns; s++)
        for (int q = S.child_ptr[s]; q < S.child_ptr[s + 1]; q++) {
            const int ch = S.child_list[q];
            int* sl = slot.data() + slot_off[s] + static_cast<long long>(q - S.child_ptr[s]) * S.nrow[s];
            for (long long j = S.relind_off[ch]; j < S.relind_off[ch + 1]; j++)
                sl[S.relind[j]] = static_cast<int>(S.upd_off[ch] / 3 + (j - S.relind_off[ch]));
        }
    // Solve items above the cut: forward sweep by level (leaves first),
    // backward sweep by level (root first).  A tile holds about lev_td doubles
    // of M: a level's share per resident CTA, so that levels with little work
    // still spread over the chip, within [kTileMin, kTileMax] (below it the
    // tiles' repeated assembly of f costs more than the spread gives, above it
    // a level's last tiles run alone).
    EFEM_CUDA(cudaFuncSetAttribute(k_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSolveSmem)));
    int per_sm = 0, sms = 0;
    EFEM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_solve, kST, kSolveSmem));
    EFEM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m.device));
    P.slots = std::max(1, per_sm) * std::max(1, sms);
    std::vector<int> lev_td(nlev, 0);
    auto area = [&](int s) { return static_cast<long long>(S.nrow[s]) * S.ncol[s]; };
    for (int l = 0; l < nlev; l++) {
        long long sum = 0;
        for (int q = S.level_ptr[l]; q < S.level_ptr[l + 1]; q++) sum += area(S.level_list[q]);
        lev_td[l] = static_cast<int>(std::min<long long>(kTileMax, std::max<long long>(kTileMin, sum / P.slots)));
    }
    auto fwd_rows = [&](int s) {  // rows of a forward tile: equal tiles of about lev_td doubles, a multiple of 8
        const int r = S.nrow[s], td = lev_td[lev[s]];
        const long long nt = std::max<long long>(std::max<long long>(1, (area(s) + td / 2) / td), (r + kMaxR - 1) / kMaxR);
        return std::min(kMaxR, std::max(8, static_cast<int>(((r + nt - 1) / nt + 7) / 8 * 8)));
    };
    auto bwd_cols = [&](int s) {  // columns of a backward tile, a multiple of 4
        const int c = S.ncol[s], td = lev_td[lev[s]];
        const long long nt = std::max<long long>(1, (area(s) + td / 2) / td);
        return std::min(32, std::max(4, static_cast<int>(((c + nt - 1) / nt + 3) / 4 * 4)));
    };
    std::vector<int> tY(S.ns, 0), tG(S.ns, 0), tX(S.ns, 0);  // tiles that complete y, the children's g, x of a front
    for (int s = 0; s < S.ns; s++) {
        const int c = S.ncol[s], r = S.nrow[s], fr = fwd_rows(s), bc = bwd_cols(s);
        tY[s] = (c + fr - 1) / fr;
        tX[s] = (c + bc - 1) / bc;
        if (S.parent[s] >= 0 && !in_sub[s])  // (subtree roots finish before k_solve)
            tG[S.parent[s]] += (r + fr - 1) / fr - c / fr;
    }
    std::vector<SolveItem> items;
    auto sweep = [&](int l, bool fwd) {
        for (int q = S.level_ptr[l]; q < S.level_ptr[l + 1]; q++) {
            const int s = S.level_list[q], p = S.parent[s];
            const int n = fwd ? S.nrow[s] : S.ncol[s], step = fwd ? fwd_rows(s) : bwd_cols(s);
            for (int o = 0; o < n; o += step)
                items.push_back(SolveItem { fwd ? kFwdTile : kBwdTile, s, o, std::min(n, o + step), p, S.nrow[s], S.ncol[s],
                    S.first[s], S.child_ptr[s + 1] - S.child_ptr[s], fwd ? tG[s] : tY[s], !fwd && p >= 0 ? tX[p] : 0, 0,
                    xw_off[s], S.rows_off[s], slot_off[s], S.upd_off[s] });
        }
    };
    for (int l = K; l < nlev; l++) sweep(l, true);
    for (int l = nlev - 1; l >= K; l--) sweep(l, false);
    P.n_items = static_cast<int>(items.size());
    P.h_item_front.resize(items.size());
    for (size_t i = 0; i < items.size(); i++) P.h_item_front[i] = items[i].s;
    P.solve_smem = kSolveSmem;
    // node index in v of every front row
    std::vector<int> prow(S.rows.size());
    for (size_t q = 0; q < S.rows.size(); q++) prow[q] = S.perm[S.rows[q]];
    // device arrays
    efem_status st;
#define UP(p, v)                                       \
    if ((st = dev_upload(&(p), (v))) != EFEM_OK) return st;
    UP(P.d_first, S.first);
    UP(P.d_ncol, S.ncol);
    UP(P.d_nrow, S.nrow);
    UP(P.d_child_ptr, S.child_ptr);
    UP(P.d_child_list, S.child_list);
    UP(P.d_relind, S.relind);
    UP(P.d_perm, S.perm);
    UP(P.d_front_off, S.front_off);
    UP(P.d_rows_off, S.rows_off);
    UP(P.d_relind_off, S.relind_off);
    UP(P.d_xw_off, xw_off);
    UP(P.d_level_list, S.level_list);
    UP(P.d_slot, slot);
    UP(P.d_slot_off, slot_off);
    UP(P.d_zero, zeros);
    UP(P.d_upd_off, S.upd_off);
    UP(P.d_a_pos, S.a_pos);
    UP(P.d_a_src, S.a_src);
    UP(P.d_vals, vals);
    UP(P.d_parent, S.parent);
    UP(P.d_prow, prow);
    UP(P.d_items, items);
    if (P.n_subs > 0) {
        UP(P.d_subs, subs);
        UP(P.d_chunks, chunks);
        UP(P.d_depth, sdepth);
        UP(P.d_xidx, xidx);
    }
    UP(P.d_wtiles, wtiles);
    UP(P.d_ea, ea);
    UP(P.d_steps, steps);
    UP(P.d_invs, invs);
#undef UP
    const size_t n3 = 3 * static_cast<size_t>(std::max(S.n, 1));
    if ((st = dev_alloc(&P.d_front, static_cast<size_t>(S.front_size))) != EFEM_OK) return st;
    if ((st = dev_alloc(&P.d_xw, static_cast<size_t>(std::max<long long>(xw_size, 1)))) != EFEM_OK) return st;
    if ((st = dev_alloc(&P.d_lp, static_cast<size_t>(std::max<long long>(xw_size, 1)))) != EFEM_OK) return st;
    EFEM_CUDA(cudaMemsetAsync(P.d_xw, 0, sizeof(double) * std::max<long long>(xw_size, 1), m.stream));  // above X's diagonal, pad rows
    if ((st = dev_alloc(&P.d_upd, static_cast<size_t>(std::max<long long>(S.upd_size, 1)))) != EFEM_OK) return st;
    if ((st = dev_alloc(&P.d_y, n3)) != EFEM_OK) return st;
    if ((st = dev_alloc(&P.d_cnt, 4 * static_cast<size_t>(S.ns) + 2)) != EFEM_OK) return st;
    if ((st = dev_alloc(&P.d_fail, 1)) != EFEM_OK) return st;
    // persistent solve: as many CTAs as fit on the device at once
    P.solve_grid_full = std::max(1, std::min(P.n_items, P.slots));
    P.solve_grid = solve_grid_for(P);
    if (P.n_subs > 0) {
        EFEM_CUDA(cudaFuncSetAttribute(k_sub_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        EFEM_CUDA(cudaFuncSetAttribute(k_sub_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    }
    EFEM_CUDA(cudaStreamCreateWithFlags(&P.capture, cudaStreamNonBlocking));
    EFEM_CUDA(cudaStreamCreateWithFlags(&P.capture2, cudaStreamNonBlocking));
    EFEM_CUDA(cudaHostAlloc(&P.h_flag, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable));
    *P.h_flag = 0;
    if ((st = dev_alloc(&P.d_res, 1)) != EFEM_OK) return st;
    EFEM_CUDA(cudaMemsetAsync(P.d_res, 0, sizeof(int), m.stream));
    EFEM_CUDA(cudaMemsetAsync(P.d_cnt, 0, sizeof(int) * (4 * static_cast<size_t>(S.ns) + 2), m.stream));
    P.ready = true;  // analysed; the numeric factor follows
    return precond_factor(m, ok, ms_factor);
}

// Numeric factorisation (every solve, like LBFGSSolver::updateApproxJacobi):
// scatter L into the fronts, factor level by level, invert the diagonal blocks.
// the launches of one numeric factorisation, in order, on stream st; returns
// the number of kernels
static long long enqueue_factor(Precond& P, cudaStream_t st, cudaStream_t st2, cudaEvent_t ev)
{
    const Symbolic& S = P.S;
    long long n = 0;
    bool forked = false;
    cudaMemsetAsync(P.d_fail, 0, sizeof(int), st);
    if (P.n_zero > 0) k_zero<<<P.n_zero, kFT, 0, st>>>(P.d_front, P.d_zero);
    const long long na = static_cast<long long>(S.a_pos.size());
    k_scatter_a<<<static_cast<int>(std::min<long long>(8 * kSMs, (na + 255) / 256 + 1)), 256, 0, st>>>(
        P.d_front, P.d_a_pos, P.d_a_src, P.d_vals, na);
    n += 2;
    FrontArgs a = args_of(P);
    auto fork = [&]() {  // the second branch goes on from here
        cudaEventRecord(ev, st);
        cudaStreamWaitEvent(st2, ev, 0);
        forked = true;
    };
    for (int l = 0; l < P.nlev; l++) {
        const int cnt = P.ea_off[l + 1] - P.ea_off[l];
        if (cnt > 0) {
            launch_k(k_extend_add, cnt, kFT, 0, st, a, static_cast<const int4*>(P.d_ea + P.ea_off[l]));
            n++;
        }
        launch_k(k_diag, S.level_ptr[l + 1] - S.level_ptr[l], kFT, 0, st, a, static_cast<const int*>(P.d_level_list + S.level_ptr[l]));
        n++;
        // the steps; beside them, and beside the levels above, X and W
        int iv = P.lev_first_inv[l];
        const int s0 = P.lev_first_step[l], s1 = P.lev_first_step[l + 1], nw = P.w_off[l + 1] - P.w_off[l];
        for (int q = s0; q < s1; q++) {
            if (P.steps[q].cnt > 0) launch_k(k_step, P.steps[q].cnt, kFT, 0, st, a, static_cast<const int4*>(P.d_steps + P.steps[q].off), P.steps[q].k0);
            n++;
            const bool more = iv < P.lev_first_inv[l + 1] && P.invs[iv].after == q - s0;
            if (more || (q == s1 - 1 && nw > 0)) fork();
            for (; iv < P.lev_first_inv[l + 1] && P.invs[iv].after == q - s0; iv++, n++)
                k_inverse<<<P.invs[iv].cnt, 256, 0, st2>>>(a, P.d_invs + P.invs[iv].off, P.invs[iv].h, P.invs[iv].second);
        }
        if (nw > 0) {
            k_w<<<nw, 256, 0, st2>>>(a, P.d_wtiles + P.w_off[l]);
            n++;
        }
    }
    if (forked) {
        cudaEventRecord(ev, st2);
        cudaStreamWaitEvent(st, ev, 0);
    }
    return n;
}

// The factorisation's few hundred dependent launches are captured once into a
// CUDA graph and replayed every solve (shorter gaps between the launches).
static efem_status precond_factor(Model& m, int* ok, double* ms_factor)
{
    Precond& P = *m.precond;
    if (!P.factor_exec) {
        std::lock_guard<std::mutex> lock(capture_mutex());
        // with programmatic dependent launch along the steps; a capture that refuses it is made with plain launches
        for (int attempt = 0; attempt < 2 && !P.factor_exec; attempt++) {
            cudaGraph_t g = nullptr;
            cudaEvent_t ev;
            EFEM_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
            cudaError_t e = cudaStreamBeginCapture(P.capture, cudaStreamCaptureModeThreadLocal);
            if (e == cudaSuccess) {
                t_pdl = attempt == 0;
                P.factor_launches = enqueue_factor(P, P.capture, P.capture2, ev);
                t_pdl = false;
                e = cudaStreamEndCapture(P.capture, &g);
            }
            cudaEventDestroy(ev);
            if (e == cudaSuccess) e = cudaGraphInstantiate(&P.factor_exec, g, 0);
            if (g) cudaGraphDestroy(g);
            if (e != cudaSuccess) {
                P.factor_exec = nullptr;
                cudaGetLastError();
                if (attempt == 0) continue;
                set_error(std::string("factorisation graph: ") + cudaGetErrorString(e));
                return EFEM_ERR_CUDA;
            }
        }
    }
    cudaEvent_t e0, e1;
    EFEM_CUDA(cudaEventCreate(&e0));
    EFEM_CUDA(cudaEventCreate(&e1));
    EFEM_CUDA(cudaEventRecord(e0, m.stream));
    EFEM_CUDA(cudaGraphLaunch(P.factor_exec, m.stream));
    m.launches += P.factor_launches;
    EFEM_CUDA(cudaGetLastError());
    EFEM_CUDA(cudaEventRecord(e1, m.stream));
    int fail = 0;
    EFEM_CUDA(cudaMemcpyAsync(&fail, P.d_fail, sizeof(int), cudaMemcpyDeviceToHost, m.stream));
    EFEM_CUDA(cudaStreamSynchronize(m.stream));
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    P.ms_factor = ms;
    P.ok = fail == 0;
    P.factored = true;
    *ok = P.ok;
    *ms_factor = ms;
    return EFEM_OK;
}

void precond_drop_graphs(Model& m)
{
    if (!m.precond) return;
    m.epoch++;  // the solver's iteration graphs hold the persistent solve's arguments
}

efem_status precond_sync_grid(Model& m)
{
    if (!m.precond || !m.precond->ready) return EFEM_OK;
    Precond& P = *m.precond;
    const int want = solve_grid_for(P);
    if (want == P.solve_grid) return EFEM_OK;
    P.solve_grid = want;
    m.epoch++;  // the solver's iteration graphs hold the old grid
    return EFEM_OK;
}

efem_status precond_apply(Model& m, double* d_v)
{
    efem_status s = precond_enqueue(m, d_v, m.stream);
    if (s == EFEM_OK) m.launches += precond_launch_count(m);
    return s;
}

efem_status precond_enqueue(Model& m, double* d_v, cudaStream_t stream, unsigned long long* stamp)
{
    if (!m.precond || !m.precond->factored || !m.precond->ok) {
        set_error("preconditioner not factored");
        return EFEM_ERR_ARG;
    }
    Precond& P = *m.precond;
    if (P.S.n == 0) return EFEM_OK;
    const efem_status s = enqueue_solve(P, args_of(P), SolveBufs { P.d_y, P.d_upd, P.d_cnt }, d_v, stream, wait_cfg(m), true, stamp);
    if (m.opts.wait_test == 2) m.opts.wait_test = 0;  // that was the one application
    if (s != EFEM_OK) return s;
    EFEM_CUDA(cudaGetLastError());
    return EFEM_OK;
}

efem_status precond_set_groups(Model& m, const std::vector<int>& group_of_free_node, const int* d_frozen)
{
    if (!m.precond || !m.precond->ready) {
        set_error("precond_set_groups: no solve schedule");
        return EFEM_ERR_ARG;
    }
    Precond& P = *m.precond;
    if (P.n_subs > 0) return EFEM_OK;  // subtree solves do not skip; leave the schedule as it is
    std::vector<int> g(std::max(1, P.n_items), 0);
    for (int i = 0; i < P.n_items; i++) {
        const int s = P.h_item_front[i];
        g[i] = group_of_free_node[P.S.perm[P.S.first[s]]];
    }
    dev_free(P.d_item_group);
    efem_status st = dev_upload(&P.d_item_group, g);
    if (st != EFEM_OK) return st;
    P.d_frozen = d_frozen;
    m.epoch++;  // captured solves hold the old arguments
    return EFEM_OK;
}

bool precond_has_groups(const Model& m) { return m.precond && m.precond->d_item_group; }

long long precond_launch_count(const Model& m)
{
    if (!m.precond) return 0;
    return (m.precond->n_items > 0 ? 1 : 0) + (m.precond->n_subs > 0 ? 2 : 0);
}

const int* precond_error_flag(const Model& m) { return m.precond ? m.precond->d_res : nullptr; }

efem_status precond_gave_up(Model& m)
{
    if (m.precond && m.precond->h_flag) *static_cast<volatile int*>(m.precond->h_flag) = 0;
    set_error("the triangular solve of the preconditioner gave up waiting for a front");
    return EFEM_ERR_TIMEOUT;
}

efem_status precond_check(Model& m)
{
    if (!m.precond || !m.precond->h_flag) return EFEM_OK;
    EFEM_CUDA(cudaStreamSynchronize(m.stream));
    return *static_cast<volatile int*>(m.precond->h_flag) ? precond_gave_up(m) : EFEM_OK;
}

// ============================================================================
// Allocation-free H0 application.
//
// Some callers cannot call cudaMalloc at the moment they need H0 v: code that
// runs while a CUDA stream capture is open (cudaMalloc is not allowed there),
// code inside another framework's allocator (a caching allocator that owns the
// device's free memory and must not see foreign allocations), or real-time
// control loops that forbid the implicit device synchronisation an allocation
// can cause.  For them efem_precond_apply_noalloc runs the same forward and
// backward sweeps as efem_precond_apply, but its working memory (the forward
// result, 3 per free node, the fronts' update vectors, and the solve's
// completion counters) lives in the fixed array below instead of buffers owned
// by the model.
//
// Limits and sharing:
//   * the array holds kNoAllocDoubles doubles (16 MiB); a model that needs
//     more than that by the interface's formula (6 * free nodes + its
//     update-vector length + 2 * fronts + 1) is rejected.  The sweeps use
//     half of the formula's first term; which models are refused is part of
//     the interface and stays;
//   * every GPU that loads this library keeps the array until the process
//     exits;
//   * all calls share the array and it keeps the last call's contents; the
//     counters are cleared by each call and every other entry is written
//     before it is read, but calls that overlap on the GPU (other streams, other threads, other
//     models) race on it and must be serialised by the caller.
// ============================================================================
namespace {
constexpr size_t kNoAllocDoubles = size_t(2) << 20;
static __device__ __align__(256) double g_noalloc_scratch[kNoAllocDoubles];

// device address of g_noalloc_scratch, looked up once per device; in host
// code the array's name is only a host-side stand-in, never a device address
std::mutex g_noalloc_mutex;
double* g_noalloc_addr[256] = {};

efem_status noalloc_scratch(int device, double** out)
{
    if (device < 0 || device >= 256) {
        set_error("device ordinal out of range for the static workspace");
        return EFEM_ERR_ARG;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_addr[device]) {
        EFEM_CUDA(cudaSetDevice(device));
        void* p = nullptr;
        EFEM_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
        g_noalloc_addr[device] = static_cast<double*>(p);
    }
    *out = g_noalloc_addr[device];
    return EFEM_OK;
}
}  // namespace

}  // namespace efem

extern "C" efem_status efem_precond_apply_noalloc(void* model, double* d_v)
{
    using namespace efem;
    if (!model || !d_v) {
        set_error("null model or vector");
        return EFEM_ERR_ARG;
    }
    Model& m = *static_cast<Model*>(model);
    // by the interface's formula 6 per free node are the least any model needs: refuse
    // models that cannot fit before asking for anything else
    if (6 * static_cast<size_t>(m.n_free) > kNoAllocDoubles) {
        set_error("model needs at least " + std::to_string(6 * static_cast<size_t>(m.n_free))
            + " doubles of workspace; the static workspace of efem_precond_apply_noalloc holds "
            + std::to_string(kNoAllocDoubles));
        return EFEM_ERR_ARG;
    }
    if (!m.on_device || !m.precond || !m.precond->factored || !m.precond->ok) {
        set_error("efem_precond_apply_noalloc needs an existing positive-definite factor: call efem_solve or "
                  "efem_precond_apply once first");
        return EFEM_ERR_ARG;
    }
    Precond& P = *m.precond;
    const Symbolic& S = P.S;
    const size_t n3 = 3 * static_cast<size_t>(S.n);
    const size_t n_cnt = 4 * static_cast<size_t>(S.ns) + 2;
    const size_t need = 2 * n3 + static_cast<size_t>(S.upd_size) + (n_cnt + 1) / 2;
    if (need > kNoAllocDoubles) {
        set_error("model needs " + std::to_string(need) + " doubles of workspace; the static workspace of "
            "efem_precond_apply_noalloc holds " + std::to_string(kNoAllocDoubles));
        return EFEM_ERR_ARG;
    }
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    EFEM_CUDA(cudaStreamIsCapturing(m.stream, &cs));
    const bool capturing = cs != cudaStreamCaptureStatusNone;
    double* scratch = nullptr;
    if (capturing) {  // only a cached address: no CUDA runtime call that a capture forbids
        std::lock_guard<std::mutex> lock(g_noalloc_mutex);
        scratch = m.device >= 0 && m.device < 256 ? g_noalloc_addr[m.device] : nullptr;
        if (!scratch) {
            set_error("efem_precond_apply_noalloc: the first call on a device must come before any stream "
                      "capture (it looks up the static workspace's device address)");
            return EFEM_ERR_ARG;
        }
    } else {
        efem_status st = noalloc_scratch(m.device, &scratch);
        if (st != EFEM_OK) return st;
        EFEM_CUDA(cudaSetDevice(m.device));
    }
    if (S.n == 0) return EFEM_OK;
    // This thread's host-side calls below (pointer check, flag read) must not
    // invalidate a capture that the caller has open on some other stream.
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    EFEM_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
    struct Restore {
        cudaStreamCaptureMode mode;
        ~Restore() { cudaThreadExchangeStreamCaptureMode(&mode); }
    } restore { mode };
    if (!capturing) {  // d_v must be memory this GPU addresses (not checked while capturing)
        cudaPointerAttributes a {};
        const bool ok = cudaPointerGetAttributes(&a, d_v) == cudaSuccess
            && (a.type == cudaMemoryTypeManaged || (a.type == cudaMemoryTypeDevice && a.device == m.device)
                || (a.type == cudaMemoryTypeHost && a.devicePointer != nullptr));
        if (!ok) {
            cudaGetLastError();
            set_error("d_v is not device memory of the model's GPU");
            return EFEM_ERR_ARG;
        }
    }
    int* counters = reinterpret_cast<int*>(scratch + n3 + S.upd_size);
    const SolveBufs b { scratch, scratch + n3, counters };
    efem_status st = enqueue_solve(P, args_of(P), b, d_v, m.stream, wait_cfg(m), false);
    if (st != EFEM_OK) return st;
    EFEM_CUDA(cudaGetLastError());
    if (capturing) return EFEM_OK;  // recorded into the caller's graph; a give-up shows as NaN in d_v
    int flag = 0;
    EFEM_CUDA(cudaMemcpyAsync(&flag, counters + 4LL * S.ns + 1, sizeof(int), cudaMemcpyDeviceToHost, m.stream));
    EFEM_CUDA(cudaStreamSynchronize(m.stream));
    return flag ? precond_gave_up(m) : EFEM_OK;
}
