// bx_graph.cu -- BETSE's cell-network Poisson operators at any cluster size.
//
// Cells.graphLaplacian (betse/science/cells.py:1845-1894) forms, from the
// incidence matrix D of the cluster's triangulation (one row per edge),
//     lapGJinv = pinv(D) diag(tri_len / vor_len) (-pinv(D)^T) diag(vor_sa)
//              = -L+ Lw L+ A,
// with L = D^T D the graph Laplacian, L+ its pseudo-inverse (pinv(D) =
// L+ D^T for a connected graph), Lw = D^T diag(tri_len / vor_len) D and
// A = diag(vor_sa); physics/pressures.py:59 applies it with np.dot.  BETSE
// builds it densely with an SVD, O(n^3); here L+ is applied to a block of
// right-hand sides by conjugate gradients in FP64, one independent CG per
// column, preconditioned by an aggregation multigrid V-cycle:
//   * level l+1 aggregates consecutive groups of four nodes of level l
//     (node i -> i / 4); the caller orders the cells so that consecutive
//     cells are neighbours (the generator's Z curve), and passes each
//     level's Galerkin operator P^T L P (again a graph Laplacian);
//   * one damped Jacobi sweep (omega 0.9: the spectrum of D^-1 L ends at 2)
//     before and after the coarse correction, which is over-weighted by 1.8
//     (unsmoothed aggregation under-corrects smooth errors);
//   * the first level of at most 512 nodes is solved exactly with its
//     pseudo-inverse, built on the GPU at creation (with 2048 nodes 76 CG
//     iterations instead of 88, but 30 ms more at creation); in blocks of more
//     than eight columns, which the FP64 pipe bounds, the first level whose
//     dense product stays under 4 % of the work (its nodes squared at most
//     twice the finest level's); a graph of at most 512 nodes is that one
//     product in any block (4 iterations instead of 36);
//   * every right-hand side and every preconditioned residual is projected
//     orthogonal to the constants (the null space of L), so the iterate
//     stays in the range of L+.
// At 100k cells this takes 84 iterations to a relative residual of 1e-12, 88 to
// 0.4 of it, where a solve to 1e-12 stops (two sweeps on each side and a 64-node
// coarsest level: 76 to 1e-12; plain Jacobi-preconditioned CG: ~1500).
//
// A solve is one cooperative launch (k_graph_cg), one CTA per SM, whose phases
// (product, update, a restriction and a prolongation per level, the dense
// level, the last sweep) meet at a bounded grid barrier of 1.3 us.  As separate
// launches an iteration at 100k cells and one column was 36 kernels and 0.3 ms;
// it is 50 us now, about 10 us of it FP64 work and 14 us barriers, the rest the
// L2 round trips of the phases.  lapGJinv X (two solves to 1e-12), ms, separate
// launches -> one launch: 100k cells, 1 / 16 / 64 / 256 columns 46.4 -> 9.0,
// 87 -> 48, 233 -> 137, 852 -> 505; 20k cells 29.0 -> 4.8, 32.3 -> 15.9, 54.1 ->
// 29.5, 151 -> 91; 5k cells, one column 21.1 -> 3.0.  Wide blocks are bound by
// the FP64 pipe: one sweep instead of two on each side, s = omega D^-1 b kept
// beside b and the prolongation folded into the sweep above it leave 45 FP64
// instructions a node and column of about 100.
//
// Layout: every block of vectors is [n][nrhs] row-major (the nrhs values of
// a node contiguous).  Column sums are deterministic (fixed partition, fixed
// order) and every CTA adds the same CTA partials, so all of them take the
// same decisions.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/bx.h"
#include "bx_sync.cuh"

void bx_record_error(const char* msg);

namespace {

constexpr int kAgg = 4;             // nodes per aggregate
constexpr double kOmega = 0.9;
constexpr double kCoarseWeight = 1.8;
constexpr int kMaxLevels = 16;
constexpr int kDense = 512;         // most nodes of the dense level
constexpr int kNarrow = 8;          // columns of a narrow block
constexpr int kCgT = 768;           // threads per CTA of the solver (85 registers each)
constexpr int kCheckEvery = 4;      // iterations between residual checks
// A solve whose columns the caller gets stops at this part of the tolerance.  With
// one sweep on each side the residual falls in smaller steps than with two, so the
// check that finds it below the tolerance finds it less far below, and the error
// follows.  lapGJinv X at tol 1e-12 against 64 bits (1e-13, means of four blocks of
// 1 / 4 / 16 columns): two sweeps | one, stopping at tol | at 0.4 tol
//   95,800 cells  6.1 / 5.0 / 4.8 | 9.6 / 9.2 / 7.3 | 1.8 / 1.8 / 1.6
//   60,000 cells   18 /  11 / 3.6 | 7.3 / 7.3 / 5.5 | 5.9 / 3.4 / 1.4
//   20,000 cells   18 / 7.7 / 4.0 | 5.3 / 5.2 / 8.5 | 5.3 / 5.2 / 1.5
//    3,000 cells  4.3 / 4.3 / 5.2 | 1.4 / 1.3 / 1.0 | the same
// It costs up to four iterations: 95,800 cells 8.53 -> 8.93 ms, 20,000 cells 4.77
// either way.  (The dense operator's columns are rounded to BF16 pairs: it keeps the
// tolerance itself.)
constexpr double kStopAt = 0.4;
constexpr int kSharedRhs = 64;      // widest block whose column scalars sit in shared memory
constexpr size_t kStageMax = 192 * 1024;   // shared memory for matrix rows
constexpr long long kBarrierNs = 2000000000LL;

int gfail(int code, const std::string& msg) {
  bx_record_error(msg.c_str());
  return code;
}

#define GCK(call)                                                                          \
  do {                                                                                     \
    cudaError_t e_ = (call);                                                               \
    if (e_ != cudaSuccess) return gfail(BX_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// Kernels over [rows][K] blocks: a CTA covers kt columns (a power of two up
// to 256, so that wide blocks read long runs of each row) times 256 / kt
// rows, and strides over the rows.
struct Shape {
  dim3 grid, block;
};

Shape shape_for(int rows, int K) {
  int kt = 1;
  while (kt < K && kt < 256) kt <<= 1;
  const int rpb = 256 / kt;
  const int gx = (K + kt - 1) / kt;
  // about 16 CTAs per SM in all, each striding over rows: short-lived CTAs
  // of one row each cost more to schedule than their work
  const int gy = std::max(1, std::min((rows + rpb - 1) / rpb, std::max(1, 152 * 16 / gx)));
  return {dim3((unsigned)gx, (unsigned)gy), dim3((unsigned)kt, (unsigned)rpb)};
}

#define FOR_RC(rows, K)                                       \
  const int k = blockIdx.x * blockDim.x + threadIdx.x;        \
  if (k >= (K)) return;                                       \
  for (int i = blockIdx.y * blockDim.y + threadIdx.y; i < (rows); i += gridDim.y * blockDim.y)

#define LAUNCH(kern, rows, K, s, ...)                          \
  do {                                                        \
    const Shape sh_ = shape_for((rows), (K));                 \
    kern<<<sh_.grid, sh_.block, 0, (s)>>>(__VA_ARGS__);       \
  } while (0)

// sum over row i's entries p of val[p] * xv(col[p]), in entry order
template <class F>
__device__ __forceinline__ double row_dot(const int* __restrict__ ptr, const int* __restrict__ col,
                                          const double* __restrict__ val, int i, F xv) {
  double sum = 0.0;
  for (int p = ptr[i]; p < ptr[i + 1]; ++p) sum += val[p] * xv(col[p]);
  return sum;
}

// out = L in (CSR, rows of K values)
__global__ void k_spmv(int n, int K, const int* __restrict__ ptr, const int* __restrict__ col,
                       const double* __restrict__ val, const double* __restrict__ in, double* __restrict__ out) {
  FOR_RC(n, K) {
    out[(long long)i * K + k] = row_dot(ptr, col, val, i, [&](int j) { return in[(long long)j * K + k]; });
  }
}

// Y = sign * diag(s) X (s null: 1)
__global__ void k_row_scale(int n, int K, const double* __restrict__ s, const double* __restrict__ X,
                            double* __restrict__ Y, double sign) {
  FOR_RC(n, K) Y[(long long)i * K + k] = sign * (s ? s[i] : 1.0) * X[(long long)i * K + k];
}

// the scaled identity columns col0 .. col0+K-1: E[i][k] = s_i where i == col0 + k
__global__ void k_scaled_identity(int n, int K, int col0, const double* __restrict__ s, double* __restrict__ E) {
  FOR_RC(n, K) E[(long long)i * K + k] = (i == col0 + k) ? s[i] : 0.0;
}

// One level as the solver reads it.
struct CgLevel {
  int n;
  int r0;                  // row of ptr[0] and dinv[0] (staged: the CTA's first; entries then count from there too)
  const int *ptr, *col;
  const double *val, *dinv;
  double *b, *s, *x;       // right-hand side, omega D^-1 b, s + w_c * prolonged correction
};

struct CgArgs {
  int K, lc;               // columns; index of the dense level
  int G;                   // column groups: CTA b has row block b / G of the slabs b % G, b % G + G, ...
  int staged;              // levels [staged, lc) keep this CTA's matrix rows in shared memory
  CgLevel lv[kMaxLevels];
  const double* dense;     // [lv[lc].n]^2
  const double* B;
  double *X, *R, *Z, *P0, *P1, *Q;
  double* part;            // [2][3][grid][K] CTA partials of a phase's column sums
  double* scal;            // [grid][8][K] this CTA's column scalars: r.z twice, |b|^2, mean, factor, then three totals
  double tol;
  int max_iter;
  unsigned* ctl;           // barrier counter, timeout flag
  double* worst;           // [8] worst relative residual of each group's columns
  double* out;             // {iterations, worst relative residual}
};

// The solver's CTA: thread t holds column t % kt (kt a power of two, 1 to 32)
// of row t / kt; wider blocks go in slabs of 32 columns, dealt to G groups of
// CTAs, so that a CTA keeps many rows a slab (one group: a 5,000-node cluster
// left 33 rows a CTA, 1.4 passes of its 24 row lanes).
//
// Every barrier's acquire empties the SM's L1, so the matrix rows of a CTA sit in
// shared memory: from global memory each phase waited for three dependent L2
// round trips (row pointer, column, neighbour's value) instead of one.
//
// ONE: one group, so that its columns are all of them (one column, 100,043 cells:
// 9.24 ms an apply with the group's columns counted, 8.99 without).
template <bool ONE>
struct CgCta {
  const CgArgs& a;
  const CgLevel* lv;       // shared: the levels, staged rows in place of the global ones
  double* red;             // shared: [3][kCgT]
  double* sub;             // shared: [3][4][32]
  int* flag;               // shared
  int kt, col, row, rows;  // rows: rows per pass
  int kl, kown;            // log2 kt; columns of this group's slabs (some past K in the last one)
  int nrb, rb, group;      // row blocks, this CTA's row block and column group
  unsigned round;          // barriers passed
  double* scal;
  bool ok;

  __device__ CgCta(const CgArgs& args, const CgLevel* lv_, double* red_, double* sub_, double* scal_, int* flag_)
      : a(args), lv(lv_), red(red_), sub(sub_), flag(flag_), round(0), ok(true) {
    kt = 1;
    kl = 0;
    while (kt < a.K && kt < 32) kt <<= 1, ++kl;
    col = threadIdx.x & (kt - 1);
    row = threadIdx.x / kt;
    rows = kCgT / kt;
    nrb = (int)gridDim.x / a.G;
    rb = (int)blockIdx.x / a.G;
    group = (int)blockIdx.x % a.G;
    kown = ONE ? a.K : ((a.K + kt - 1) / kt - group + a.G - 1) / a.G * kt;
    scal = a.K <= kSharedRhs ? scal_ : a.scal + (size_t)blockIdx.x * 8 * a.K;
  }
  // row block b of nb of n rows, whole aggregates
  __host__ __device__ static void rows_of(int n, int nb, int b, int& lo, int& hi) {
    const int per = ((n + nb - 1) / nb + kAgg - 1) / kAgg * kAgg;
    lo = n < b * per ? n : b * per;
    hi = n < lo + per ? n : lo + per;
  }
  __device__ void range(int n, int& lo, int& hi) const { rows_of(n, nrb, rb, lo, hi); }
  // column q of this group's slabs (past K: none)
  __device__ int own(int q) const { return ONE ? q : (group + (q >> kl) * a.G) * kt + (q & (kt - 1)); }
  // the levels into `to`, the matrix rows of the staged ones into `sm`
  __device__ static void stage(const CgArgs& a, CgLevel* to, unsigned char* sm) {
    for (int l = 0; l <= a.lc; ++l) {
      CgLevel L = a.lv[l];
      if (l >= a.staged && l < a.lc) {
        int lo, hi;
        rows_of(L.n, (int)gridDim.x / a.G, (int)blockIdx.x / a.G, lo, hi);
        const int nr = hi - lo, p0 = L.ptr[lo], ne = L.ptr[hi] - p0;
        double* val = reinterpret_cast<double*>(sm);
        double* dinv = val + ne;
        int* col = reinterpret_cast<int*>(dinv + nr);
        int* ptr = col + ne;
        for (int q = threadIdx.x; q < ne; q += kCgT) {
          val[q] = L.val[p0 + q];
          col[q] = L.col[p0 + q];
        }
        for (int q = threadIdx.x; q < nr; q += kCgT) dinv[q] = L.dinv[lo + q];
        for (int q = threadIdx.x; q <= nr; q += kCgT) ptr[q] = L.ptr[lo + q] - p0;
        sm += stage_bytes(nr, ne);
        L.r0 = lo;
        L.val = val;
        L.col = col;
        L.dinv = dinv;
        L.ptr = ptr;
      }
      if (threadIdx.x == 0) to[l] = L;
    }
    __syncthreads();
  }
  __host__ __device__ static size_t stage_bytes(int nr, int ne) {
    return ((size_t)12 * ne + (size_t)12 * nr + 4 + 15) & ~(size_t)15;
  }
  __device__ bool barrier() {
    __syncthreads();
    if (threadIdx.x == 0) bx::res_arrive(a.ctl);
    ++round;
    ok = bx::res_wait(a.ctl, round * gridDim.x, kBarrierNs, flag);
    return ok;
  }
  // CTA sums of nq per-thread values of slab kb, to the partials of buffer buf
  __device__ void cta_sum(int buf, int kb, int nq, const double* v) {
    for (int q = 0; q < nq; ++q) red[q * kCgT + threadIdx.x] = v[q];
    __syncthreads();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, q = w >> 2;
    if (q < nq) {
      const int u = threadIdx.x & 127;           // 128 threads a quantity, kCgT / 128 values each
      double s = 0.0;
#pragma unroll
      for (int j = 0; j < kCgT / 128; ++j) s += red[q * kCgT + j * 128 + u];
      for (int o = 16; o >= kt; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane < kt) sub[(q * 4 + (w & 3)) * 32 + lane] = s;
    }
    __syncthreads();
    const int k = kb + (int)threadIdx.x % 32;
    const int qq = threadIdx.x / 32;
    if (qq < nq && (int)threadIdx.x % 32 < kt && k < a.K) {
      const double* p = sub + qq * 4 * 32 + threadIdx.x % 32;
      a.part[(((size_t)buf * 3 + qq) * nrb + rb) * a.K + k] = (p[0] + p[32]) + (p[64] + p[96]);
    }
    __syncthreads();
  }
  // totals of quantities 0..nq-1 of buffer buf into tot[q][k], this group's
  // columns: a warp per (quantity, column), its lanes in a fixed order
  __device__ void totals(int buf, int nq) const {
    const int lane = threadIdx.x & 31, K = a.K;
    double* tot = scal + (size_t)5 * K;
    for (int e = threadIdx.x >> 5; e < nq * kown; e += kCgT / 32) {
      const int q = e / kown, k = own(e - q * kown);
      if (!ONE && k >= K) continue;
      const double* p = a.part + ((size_t)buf * 3 + q) * nrb * K + k;
      double s = 0.0;
      for (int c0 = lane; c0 < nrb; c0 += 32 * 5) {              // 152 CTAs: one round of loads
        double x[5];
#pragma unroll
        for (int u = 0; u < 5; ++u) x[u] = __ldcg(p + (size_t)min(c0 + 32 * u, nrb - 1) * K);
#pragma unroll
        for (int u = 0; u < 5; ++u) s += c0 + 32 * u < nrb ? x[u] : 0.0;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) tot[(size_t)q * K + k] = s;
    }
    __syncthreads();
  }
  // f(k) over this group's columns, a thread each
  template <class F>
  __device__ void over_own(F f) const {
    for (int q = threadIdx.x; q < kown; q += kCgT) {
      const int k = own(q);
      if (ONE || k < a.K) f(k);
    }
    __syncthreads();
  }
  __device__ double tot(int q, int k) const { return scal[(size_t)(5 + q) * a.K + k]; }
  // f(i, k, at) over this CTA's rows of n in the current slab
  template <class F>
  __device__ void over_rows(int n, int k, F f) const {
    int lo, hi;
    range(n, lo, hi);
    for (int i = lo + row; i < hi; i += rows) f(i, (size_t)i * a.K + k);
  }
  // sum over row i's entries of val * xv(entry's column), in entry order; the
  // loads of eight entries are in flight together (a row has seven or so)
  template <class F>
  __device__ static double dot(const CgLevel& L, int i, F xv) {
    double s = 0.0;
    const int e = L.ptr[i + 1 - L.r0];
    for (int p = L.ptr[i - L.r0]; p < e; p += 8) {
      int c[8];
      double v[8], x[8];
      // past the end: this row's own value times zero, so that no load waits on a branch
#pragma unroll
      for (int u = 0; u < 8; ++u) c[u] = p + u < e ? L.col[p + u] : i;
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = xv(c[u]);
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = p + u < e ? L.val[p + u] : 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u) s += v[u] * x[u];
    }
    return s;
  }
  // level l+1: b = the aggregates' sums of (b - L s), s = omega D^-1 b
  __device__ void restrict_to(int l) const {
    const CgLevel &F = lv[l], &C = lv[l + 1];
    const bool smoothed = l + 1 < a.lc;
    const int K = a.K;
    for (int kb = group * kt; kb < K; kb += a.G * kt) {
      const int k = kb + col;
      if (kt <= 8) {
        // a lane per fine row; an aggregate's four rows are neighbours in the warp
        int lo, hi;
        range(F.n, lo, hi);
        for (int i0 = lo; i0 < hi; i0 += rows) {
          const int i = i0 + row;
          double r = 0.0;
          const bool puts = i < hi && k < K && (i & 3) == 0;
          const double wd = puts && smoothed ? kOmega * a.lv[l + 1].dinv[i >> 2] : 0.0;   // another CTA's row: not staged
          if (i < hi && k < K)
            r = __ldcg(F.b + (size_t)i * K + k) - dot(F, i, [&](int j) { return __ldcg(F.s + (size_t)j * K + k); });
          r += __shfl_xor_sync(0xffffffffu, r, kt);
          r += __shfl_xor_sync(0xffffffffu, r, 2 * kt);
          if (puts) put(C, i >> 2, k, r, smoothed, wd);
        }
      } else if (k < K) {
        int lo, hi;
        range(F.n, lo, hi);
        for (int c = (lo + kAgg - 1) / kAgg + row; c * kAgg < hi; c += rows) {   // lo: whole aggregates, or n
          double r = 0.0;
          for (int i = c * kAgg; i < min(c * kAgg + kAgg, F.n); ++i)
            r += __ldcg(F.b + (size_t)i * K + k) - dot(F, i, [&](int j) { return __ldcg(F.s + (size_t)j * K + k); });
          put(C, c, k, r, smoothed, smoothed ? kOmega * a.lv[l + 1].dinv[c] : 0.0);
        }
      }
    }
  }
  __device__ void put(const CgLevel& C, int c, int k, double r, bool smoothed, double wd) const {
    C.b[(size_t)c * a.K + k] = r;
    if (smoothed) C.s[(size_t)c * a.K + k] = wd * r;
  }
  // the correction xc of node c of level l into x of its nodes of level l-1
  __device__ void prolong(int l, int c, int k, double xc) const {
    const CgLevel& F = lv[l - 1];
    double s[kAgg];
#pragma unroll
    for (int u = 0; u < kAgg; ++u) s[u] = __ldcg(F.s + (size_t)min(c * kAgg + u, F.n - 1) * a.K + k);
#pragma unroll
    for (int u = 0; u < kAgg; ++u)
      if (c * kAgg + u < F.n) F.x[(size_t)(c * kAgg + u) * a.K + k] = s[u] + kCoarseWeight * xc;
  }
  // the dense level: sink(c, k, x) with x = dense b
  template <class F>
  __device__ void dense_solve(F sink) const {
    const CgLevel& C = lv[a.lc];
    const int n = C.n, K = a.K;
    if (K <= 4) {
      // a warp per row
      const int lane = threadIdx.x & 31, nw = kCgT / 32 * (int)gridDim.x;
      for (int c = (int)(threadIdx.x >> 5) * (int)gridDim.x + (int)blockIdx.x; c < n; c += nw) {
        const double* m = a.dense + (size_t)c * n;
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        for (int j0 = lane; j0 < n; j0 += 32 * 8) {     // eight rounds of loads in flight
          double v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) v[u] = j0 + 32 * u < n ? m[j0 + 32 * u] : 0.0;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (k >= K) break;
            double x[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) x[u] = j0 + 32 * u < n ? __ldcg(C.b + (size_t)(j0 + 32 * u) * K + k) : 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u) s[k] += v[u] * x[u];
          }
        }
        for (int k = 0; k < K; ++k) {
          double x = k == 0 ? s[0] : k == 1 ? s[1] : k == 2 ? s[2] : s[3];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
          if (lane == 0) sink(c, k, x);
        }
      }
    } else {
      // a thread per (row, column of this group), columns fastest; the warps of a
      // group's CTAs in turn, so that few rows keep every SM busy (a CTA after the
      // other: lapGJinv X of 100 nodes, 300 columns 1420 us, 1320 now)
      for (int e = (int)((threadIdx.x >> 5) * nrb + rb) * 32 + (int)(threadIdx.x & 31); e < n * kown; e += kCgT * nrb) {
        const int c = e / kown, k = own(e - c * kown);
        if (k >= K) continue;
        const double* m = a.dense + (size_t)c * n;
        double s0 = 0.0, s1 = 0.0;
        int j = 0;
        for (; j + 1 < n; j += 2) {
          s0 += m[j] * __ldcg(C.b + (size_t)j * K + k);
          s1 += m[j + 1] * __ldcg(C.b + (size_t)(j + 1) * K + k);
        }
        if (j < n) s0 += m[j] * __ldcg(C.b + (size_t)j * K + k);
        sink(c, k, s0 + s1);
      }
    }
  }
  // Z = V-cycle(R); the partials of {sum z, sum r z, sum r} go to buffer buf
  // (lv[0].b = R and lv[0].s = omega D^-1 R are written by the caller's phase)
  __device__ bool precondition(int buf) {
    const int K = a.K;
    for (int l = 0; l < a.lc; ++l) {
      restrict_to(l);
      if (!barrier()) return false;
    }
    if (a.lc == 0) {
      dense_solve([&](int c, int k, double x) { a.Z[(size_t)c * K + k] = x; });
      if (!barrier()) return false;
    } else {
      dense_solve([&](int c, int k, double x) { prolong(a.lc, c, k, x); });
      if (!barrier()) return false;
      for (int l = a.lc - 1; l > 0; --l) {
        const CgLevel& L = lv[l];
        for (int kb = group * kt; kb < K; kb += a.G * kt) {
          const int k = kb + col;
          if (k < K)
            over_rows(L.n, k, [&](int i, size_t t) {
              const double x = __ldcg(L.x + t), b = __ldcg(L.b + t);
              const double s = dot(L, i, [&](int j) { return __ldcg(L.x + (size_t)j * K + k); });
              prolong(l, i, k, x + kOmega * L.dinv[i - L.r0] * (b - s));
            });
        }
        if (!barrier()) return false;
      }
    }
    const CgLevel& L = lv[0];
    for (int kb = group * kt; kb < K; kb += a.G * kt) {
      const int k = kb + col;
      double v[3] = {0.0, 0.0, 0.0};
      if (k < K)
        over_rows(L.n, k, [&](int i, size_t t) {
          const double r = __ldcg(a.R + t);
          double z;
          if (a.lc == 0) {
            z = __ldcg(a.Z + t);
          } else {
            const double x = __ldcg(L.x + t);
            const double s = dot(L, i, [&](int j) { return __ldcg(L.x + (size_t)j * K + k); });
            z = x + kOmega * L.dinv[i - L.r0] * (r - s);
            a.Z[t] = z;
          }
          v[0] += z;
          v[1] += r * z;
          v[2] += r;
        });
      cta_sum(buf, kb, 3, v);
    }
    return barrier();
  }
};

// the larger of two values that are not negative, NaN where either is
__device__ __forceinline__ double max_or_nan(double x, double y) { return x != x || y <= x ? x : y; }

// num / den, 0 where either vanishes (a converged column stops moving)
__device__ __forceinline__ double guarded_ratio(double num, double den) {
  return (den != 0.0 && num != 0.0) ? num / den : 0.0;
}

// X = L+ B, one CTA per SM.  Per iteration:
//   P = z - mean + beta P and Q = L P (the neighbours' P formed from z and the
//   old P, so that no barrier separates the two), sum P Q;
//   X += alpha P, R -= alpha Q, omega D^-1 R, sum R R on a check;
//   the V-cycle.
template <bool ONE>
__global__ void __launch_bounds__(kCgT, 1) k_graph_cg(CgArgs a) {
  using Cta = CgCta<ONE>;
  __shared__ double red[3 * kCgT];
  __shared__ double sub[3 * 4 * 32];
  __shared__ int flag;
  __shared__ CgLevel slv[kMaxLevels];
  __shared__ double sscal[8 * kSharedRhs];
  extern __shared__ __align__(16) unsigned char staged[];
  Cta::stage(a, slv, staged);
  Cta g(a, slv, red, sub, sscal, &flag);
  const int K = a.K, n = a.lv[0].n, kt = g.kt, lane = threadIdx.x & 31;
  const CgLevel& L = slv[0];
  // column scalars: r.z of the last and of this iteration (by parity), |b|^2,
  // the mean to take off and beta or alpha.  One thread a column computes
  // them, of this group's columns: on the slow FP64 pipe every warp doing so cost
  // 7,000 cycles a phase.  (Every CTA with all columns, and the residuals in one
  // warp, lapGJinv X took, in us: 100 nodes, 1024 columns 4390, 2340 now; 700
  // nodes 24,200, 16,800 now; 1500 nodes 34,400, 26,400 now; 20,000 nodes, 256
  // columns 95,700, 91,100 now.)
  double *rz0 = g.scal, *rz1 = rz0 + K, *bb = rz1 + K, *mean = bb + K, *fac = mean + K;
  enum { BUF_Z = 0, BUF_R = 1 };   // sums that may be read while the next phase's are written

  for (int kb = g.group * kt; kb < K; kb += a.G * kt) {
    const int k = kb + g.col;
    double v = 0.0;
    if (k < K) g.over_rows(n, k, [&](int, size_t t) { v += a.B[t]; });
    g.cta_sum(BUF_Z, kb, 1, &v);
  }
  if (!g.barrier()) return;
  g.totals(BUF_Z, 1);
  g.over_own([&](int k) { mean[k] = g.tot(0, k) * (1.0 / n); });
  for (int kb = g.group * kt; kb < K; kb += a.G * kt) {
    const int k = kb + g.col;
    double v = 0.0;
    if (k < K) {
      const double m = mean[k];
      g.over_rows(n, k, [&](int i, size_t t) {
        const double r = a.B[t] - m;
        a.X[t] = 0.0;
        a.R[t] = r;
        if (a.lc > 0) L.s[t] = kOmega * L.dinv[i - L.r0] * r;
        v += r * r;
      });
    }
    g.cta_sum(BUF_R, kb, 1, &v);
  }
  if (!g.barrier()) return;
  g.totals(BUF_R, 1);
  g.over_own([&](int k) { bb[k] = g.tot(0, k); });
  if (!g.precondition(BUF_Z)) return;

  double worst = 0.0;
  int it = 1;
  for (;; ++it) {
    // ---- beta = (r.z)_new / (r.z)_old with z projected: r.(z - mean) = sum r z - mean sum r
    g.totals(BUF_Z, 3);
    const double* rzo = (it & 1) ? rz1 : rz0;
    double* rzn = (it & 1) ? rz0 : rz1;
    const bool first = it == 1;              // no old P: z with beta = 0 in its place
    const double* Po = first ? a.Z : (it & 1) ? a.P1 : a.P0;
    double* Pn = (it & 1) ? a.P0 : a.P1;
    g.over_own([&](int k) {
      const double m = g.tot(0, k) * (1.0 / n), nw = g.tot(1, k) - m * g.tot(2, k);
      mean[k] = m;
      rzn[k] = nw;
      fac[k] = first ? 0.0 : guarded_ratio(nw, rzo[k]);
    });
    for (int kb = g.group * kt; kb < K; kb += a.G * kt) {
      const int k = kb + g.col;
      double v = 0.0;
      if (k < K) {
        const double m = mean[k], be = fac[k];
        // the mean drops out of L P (L annihilates the constants)
        auto at = [&](size_t t) { return __ldcg(a.Z + t) + be * __ldcg(Po + t); };
        g.over_rows(n, k, [&](int i, size_t t) {
          const double p = at(t) - m;
          const double q = Cta::dot(L, i, [&](int j) { return at((size_t)j * K + k); });
          Pn[t] = p;
          a.Q[t] = q;
          v += p * q;
        });
      }
      g.cta_sum(BUF_R, kb, 1, &v);
    }
    if (!g.barrier()) return;
    // ---- X, R
    g.totals(BUF_R, 1);
    const bool check = it % kCheckEvery == 0 || it == a.max_iter;
    g.over_own([&](int k) { fac[k] = guarded_ratio(rzn[k], g.tot(0, k)); });
    for (int kb = g.group * kt; kb < K; kb += a.G * kt) {
      const int k = kb + g.col;
      double v = 0.0;
      if (k < K) {
        const double al = fac[k];
        g.over_rows(n, k, [&](int i, size_t t) {
          a.X[t] += al * Pn[t];
          const double r = a.R[t] - al * a.Q[t];
          a.R[t] = r;
          if (a.lc > 0) L.s[t] = kOmega * L.dinv[i - L.r0] * r;
          if (check) v += r * r;
        });
      }
      if (check) g.cta_sum(BUF_Z, kb, 1, &v);
    }
    if (!g.barrier()) return;
    if (check) {
      // the worst column, the same in every CTA (NaN if any is): the group's from
      // its totals, then the groups' across a barrier
      g.totals(BUF_Z, 1);
      double w = 0.0;
      g.over_own([&](int k) { w = max_or_nan(w, bb[k] > 0.0 ? g.tot(0, k) / bb[k] : 0.0); });
      if ((int)(threadIdx.x & ~31u) < g.kown)              // (FP64 compares are slow: warps with columns only)
        for (int o = 16; o > 0; o >>= 1) w = max_or_nan(w, __shfl_xor_sync(0xffffffffu, w, o));
      if (lane == 0) red[threadIdx.x >> 5] = w;
      __syncthreads();
      if (threadIdx.x == 0) {
        for (int q = 1; q < (min(g.kown, kCgT) + 31) / 32; ++q) w = max_or_nan(w, red[q]);   // (the other warps had no column)
        w = sqrt(w);
        red[0] = w;
        if (!ONE && g.rb == 0) a.worst[g.group] = w;
      }
      __syncthreads();
      worst = red[0];
      if (!ONE) {
        if (!g.barrier()) return;
        for (int q = 0; q < a.G; ++q) worst = max_or_nan(worst, __ldcg(a.worst + q));
      }
      __syncthreads();
      if (!(worst > a.tol) || it == a.max_iter) break;    // converged, NaN or out of iterations
    }
    if (!g.precondition(BUF_Z)) return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.out[0] = (double)it;
    a.out[1] = worst;
  }
}

// In-place Gauss-Jordan inverse of the symmetric positive definite A = L +
// (1/size of the component) on each component's block, then minus the same:
// the pseudo-inverse of the graph Laplacian L.  One cooperative launch, rows
// dealt over the CTAs, one bounded grid barrier per pivot row.
struct PinvArgs {
  int n;
  double* A;               // [n][n]
  double* piv;             // [2][n] the current pivot row
  const int* comp;         // [n] component of each node
  const double* inv_size;  // [n] 1 / its size
  unsigned* ctl;
};
__global__ void __launch_bounds__(512, 1) k_graph_pinv(PinvArgs a) {
  __shared__ int flag;
  const int n = a.n, g = gridDim.x, b = blockIdx.x, t = threadIdx.x, T = blockDim.x;
  auto proj = [&](int i, int j) { return a.comp[i] == a.comp[j] ? a.inv_size[i] : 0.0; };
  for (int i = b; i < n; i += g)
    for (int j = t; j < n; j += T) a.A[(size_t)i * n + j] += proj(i, j);
  __syncthreads();
  for (int k = 0; k < n; ++k) {
    double* pv = a.piv + (size_t)(k & 1) * n;
    if (k % g == b) {
      double* r = a.A + (size_t)k * n;
      const double d = 1.0 / r[k];
      __syncthreads();
      for (int j = t; j < n; j += T) {
        const double v = j == k ? d : r[j] * d;
        r[j] = v;
        pv[j] = v;
      }
    }
    __syncthreads();
    if (t == 0) bx::res_arrive(a.ctl);
    if (!bx::res_wait(a.ctl, (unsigned)(k + 1) * g, kBarrierNs, &flag)) return;
    for (int i = b; i < n; i += g) {
      if (i == k) continue;
      double* r = a.A + (size_t)i * n;
      const double f = r[k];
      __syncthreads();                     // every thread has read f before r[k] changes
      for (int j = t; j < n; j += T) r[j] = (j == k ? 0.0 : r[j]) - f * __ldcg(pv + j);
    }
    __syncthreads();
  }
  for (int i = b; i < n; i += g)
    for (int j = t; j < n; j += T) a.A[(size_t)i * n + j] -= proj(i, j);
}

struct Level {
  int n = 0, nnz = 0;
  int *ptr = nullptr, *col = nullptr;
  double *val = nullptr, *dinv = nullptr;
  double *x = nullptr, *s = nullptr, *b = nullptr;   // [n][max_rhs]
  double* dense = nullptr;                           // pseudo-inverse, where this level is a dense one
};

}  // namespace

struct bx_graph_solver {
  int n = 0, max_rhs = 0, grid = 0;
  int lc[2] = {0, 0};                      // the dense level of narrow (up to kNarrow columns) and wide blocks
  std::vector<size_t> stage[4];            // [level] shared memory of its staged rows, with 1, 2, 4, 8 column groups
  std::vector<Level> lv;
  int *w_ptr = nullptr, *w_col = nullptr;
  double *w_val = nullptr, *area = nullptr;
  double *R = nullptr, *Z = nullptr, *P0 = nullptr, *P1 = nullptr, *Q = nullptr, *T1 = nullptr, *T2 = nullptr;
  double *part = nullptr, *scal = nullptr, *out = nullptr;
  unsigned* ctl = nullptr;
  std::vector<void*> owned;
  ~bx_graph_solver() {
    for (void* p : owned) cudaFree(p);
  }
  template <class T>
  T* alloc(size_t n) {
    void* p = nullptr;
    if (cudaMalloc(&p, std::max<size_t>(n, 1) * sizeof(T)) != cudaSuccess) return nullptr;
    owned.push_back(p);
    return static_cast<T*>(p);
  }
};

namespace {

// X = L+ B for K columns (B and X device [n][K], distinct from the
// workspace): enqueued; slot s of `out` gets the iterations and the residual.
int solve_async(bx_graph_solver* h, const double* B, double* X, int K, double tol, int max_iter, int slot,
                cudaStream_t s, int counter = 0) {
  CgArgs a{};
  a.K = K;
  a.lc = h->lc[K > kNarrow];
  int gi = 0;                              // groups: 1, 2, 4 or 8, at most one a slab
  while (gi < 3 && (2 << gi) <= (K + 31) / 32 && (2 << gi) <= h->grid) ++gi;
  a.G = 1 << gi;
  const int grid = h->grid / a.G * a.G;
  // matrix rows in shared memory: from the coarsest level up while they fit
  size_t smem = 0;
  for (a.staged = a.lc; a.staged > 0 && smem + h->stage[gi][a.staged - 1] <= kStageMax; --a.staged)
    smem += h->stage[gi][a.staged - 1];
  for (int l = 0; l <= a.lc; ++l) {
    const Level& L = h->lv[l];
    a.lv[l] = CgLevel{L.n, 0, L.ptr, L.col, L.val, L.dinv, l == 0 ? h->R : L.b, L.s, L.x};
  }
  a.dense = h->lv[a.lc].dense;
  a.B = B; a.X = X; a.R = h->R; a.Z = h->Z; a.P0 = h->P0; a.P1 = h->P1; a.Q = h->Q;
  a.part = h->part; a.scal = h->scal; a.tol = tol; a.max_iter = max_iter; a.ctl = h->ctl + 2 * slot;
  a.out = h->out + 2 * slot;
  a.worst = h->out + 4;
  GCK(cudaMemsetAsync(a.ctl, 0, 2 * sizeof(unsigned), s));
  if (counter) GCK(cudaMemsetAsync(a.ctl, counter, sizeof(unsigned), s));
  void* args[] = {&a};
  const void* kern = a.G == 1 ? reinterpret_cast<const void*>(k_graph_cg<true>)
                              : reinterpret_cast<const void*>(k_graph_cg<false>);
  GCK(cudaLaunchCooperativeKernel(kern, dim3((unsigned)grid), dim3(kCgT), args, smem, s));
  return BX_OK;
}

// iterations and residual of the first `slots` solves (synchronises s)
int solve_result(bx_graph_solver* h, int slots, int* iters, double* rel_res, cudaStream_t s) {
  double out[4] = {0.0, 0.0, 0.0, 0.0};
  unsigned ctl[4] = {0u, 0u, 0u, 0u};
  GCK(cudaMemcpyAsync(out, h->out, sizeof(out), cudaMemcpyDeviceToHost, s));
  GCK(cudaMemcpyAsync(ctl, h->ctl, sizeof(ctl), cudaMemcpyDeviceToHost, s));
  GCK(cudaStreamSynchronize(s));
  int it = 0;
  double worst = 0.0;
  for (int q = 0; q < slots; ++q) {
    if (ctl[2 * q + 1]) return gfail(BX_ECUDA, "graph Laplacian solve: the grid barrier timed out");
    if (out[2 * q + 1] != out[2 * q + 1]) return gfail(BX_EUNSTABLE, "graph Laplacian solve: NaN residual");
    it = std::max(it, (int)out[2 * q]);
    worst = std::max(worst, out[2 * q + 1]);
  }
  if (iters) *iters = it;
  if (rel_res) *rel_res = worst;
  return BX_OK;
}

int solve(bx_graph_solver* h, const double* B, double* X, int K, double tol, int max_iter, int* iters,
          double* rel_res, cudaStream_t s) {
  const int rc = solve_async(h, B, X, K, kStopAt * tol, max_iter, 0, s);
  return rc != BX_OK ? rc : solve_result(h, 1, iters, rel_res, s);
}

// Y = lapGJinv X = -L+ Lw L+ A X
int lap_gj(bx_graph_solver* h, const double* X, double* Y, int K, double tol, int max_iter, int* iters,
           double* rel_res, cudaStream_t s, bool identity_cols = false, int col0 = 0) {
  const int n = h->n;
  if (!identity_cols) tol *= kStopAt;
  if (identity_cols)
    LAUNCH(k_scaled_identity, n, K, s, n, K, col0, h->area, h->T1);
  else
    LAUNCH(k_row_scale, n, K, s, n, K, h->area, X, h->T1, 1.0);
  int rc = solve_async(h, h->T1, h->T2, K, tol, max_iter, 0, s);
  if (rc != BX_OK) return rc;
  LAUNCH(k_spmv, n, K, s, n, K, h->w_ptr, h->w_col, h->w_val, h->T2, h->T1);
  if ((rc = solve_async(h, h->T1, h->T2, K, tol, max_iter, 1, s)) != BX_OK) return rc;
  LAUNCH(k_row_scale, n, K, s, n, K, nullptr, h->T2, Y, -1.0);
  GCK(cudaGetLastError());
  return solve_result(h, 2, iters, rel_res, s);
}

// One k_graph_pinv and its result; counter: the byte that the barrier's count starts from
int run_pinv(PinvArgs a, int grid, int counter = 0) {
  unsigned timed_out = 0;
  void* args[] = {&a};
  GCK(cudaMemset(a.ctl, 0, 2 * sizeof(unsigned)));
  if (counter) GCK(cudaMemset(a.ctl, counter, sizeof(unsigned)));
  GCK(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_graph_pinv), dim3((unsigned)std::min(a.n, grid)),
                                  dim3(512), args, 0, nullptr));
  GCK(cudaMemcpy(&timed_out, a.ctl + 1, sizeof(unsigned), cudaMemcpyDeviceToHost));
  return timed_out ? gfail(BX_ECUDA, "dense level: the grid barrier timed out") : BX_OK;
}

// The dense pseudo-inverse of a level's graph Laplacian, on the GPU.
int build_pinv(bx_graph_solver* h, Level& L, const bx_graph_level& src) {
  const int n = src.n;
  std::vector<int> root(n);
  for (int i = 0; i < n; ++i) root[i] = i;
  auto find = [&](int i) {
    while (root[i] != i) i = root[i] = root[root[i]];
    return i;
  };
  std::vector<double> A((size_t)n * n, 0.0), inv_size(n, 0.0);
  for (int i = 0; i < n; ++i)
    for (int p = src.row_ptr[i]; p < src.row_ptr[i + 1]; ++p) {
      A[(size_t)i * n + src.col[p]] += src.val[p];
      if (src.val[p] != 0.0) root[find(i)] = find(src.col[p]);
    }
  std::vector<int> comp(n), size(n, 0);
  for (int i = 0; i < n; ++i) ++size[comp[i] = find(i)];
  for (int i = 0; i < n; ++i) inv_size[i] = 1.0 / size[comp[i]];
  L.dense = h->alloc<double>((size_t)n * n);
  double *piv = nullptr, *isz = nullptr;
  int* cmp = nullptr;
  int rc = BX_OK;
  if (!L.dense || cudaMalloc(&piv, (size_t)2 * n * sizeof(double)) != cudaSuccess ||
      cudaMalloc(&isz, (size_t)n * sizeof(double)) != cudaSuccess ||
      cudaMalloc(&cmp, (size_t)n * sizeof(int)) != cudaSuccess)
    rc = gfail(BX_ENOMEM, "bx_graph_create: dense level");
  if (rc == BX_OK) {
    if (cudaMemcpy(L.dense, A.data(), A.size() * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(isz, inv_size.data(), (size_t)n * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(cmp, comp.data(), (size_t)n * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess)
      rc = gfail(BX_ECUDA, "bx_graph_create: dense level");
    else
      rc = run_pinv(PinvArgs{n, L.dense, piv, cmp, isz, h->ctl}, h->grid);
  }
  cudaFree(piv);
  cudaFree(isz);
  cudaFree(cmp);
  return rc;
}

int check_csr(const bx_graph_level& L, int n, const char* what) {
  if (L.n != n || L.nnz < 0 || !L.row_ptr || !L.col || !L.val)
    return gfail(BX_EINVAL, std::string("bx_graph_create: bad ") + what);
  if (L.row_ptr[0] != 0 || L.row_ptr[n] != L.nnz)
    return gfail(BX_EINVAL, std::string("bx_graph_create: row pointers of ") + what);
  for (int i = 0; i < n; ++i)
    if (L.row_ptr[i + 1] < L.row_ptr[i]) return gfail(BX_EINVAL, std::string("bx_graph_create: row pointers of ") + what);
  for (int p = 0; p < L.nnz; ++p)
    if (L.col[p] < 0 || L.col[p] >= n) return gfail(BX_EINVAL, std::string("bx_graph_create: column out of range in ") + what);
  return BX_OK;
}

}  // namespace

extern "C" int bx_dense_op_create_empty(int n, bx_dense_op_handle* out);
extern "C" int bx_dense_op_set_columns(bx_dense_op_handle op, int col0, int ncols, const double* cols, void* stream);
extern "C" int bx_dense_op_destroy(bx_dense_op_handle op);

extern "C" int bx_graph_create(int n_levels, const bx_graph_level* levels, const double* coarse_pinv,
                               const bx_graph_level* weighted, const double* vor_sa, int max_rhs,
                               bx_graph_handle* out) {
  if (!out || !levels || !coarse_pinv || !weighted || !vor_sa || n_levels < 1 || max_rhs < 1)
    return gfail(BX_EINVAL, "bx_graph_create: bad arguments");
  *out = nullptr;
  const int n = levels[0].n;
  if (n < 2) return gfail(BX_EINVAL, "bx_graph_create: fewer than 2 nodes");
  int rc = BX_OK;
  for (int l = 0; l < n_levels; ++l) {
    const int expect = l == 0 ? n : (levels[l - 1].n + kAgg - 1) / kAgg;
    if ((rc = check_csr(levels[l], expect, "level operator")) != BX_OK) return rc;
  }
  if ((rc = check_csr(*weighted, n, "weighted Laplacian")) != BX_OK) return rc;
  auto* h = new bx_graph_solver();
  h->n = n;
  h->max_rhs = max_rhs;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&h->grid, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    delete h;
    return gfail(BX_ECUDA, "bx_graph_create: no CUDA device");
  }
  // the dense levels (the coarsest if none is small enough)
  while (h->lc[0] < n_levels - 1 && levels[h->lc[0]].n > kDense) ++h->lc[0];
  h->lc[1] = h->lc[0];
  while (h->lc[0] > 0 && h->lc[1] < n_levels - 1 && (long long)levels[h->lc[1]].n * levels[h->lc[1]].n > 2LL * n) ++h->lc[1];
  // (a 32-bit node count is down to 512 at level 11 at the latest, and to the root
  // of twice itself sooner: whatever levels lie above, kMaxLevels holds those used)
  // shared memory of each level's staged rows: the largest row block's
  for (int gi = 0; gi < 4; ++gi)
    for (int l = 0; l < h->lc[1]; ++l) {
      const bx_graph_level& L = levels[l];
      const int nb = std::max(1, h->grid >> gi);
      size_t most = 0;
      for (int b = 0; b < nb; ++b) {
        int lo, hi;
        CgCta<true>::rows_of(L.n, nb, b, lo, hi);
        most = std::max(most, CgCta<true>::stage_bytes(hi - lo, L.row_ptr[hi] - L.row_ptr[lo]));
      }
      h->stage[gi].push_back(most);
    }
  if (cudaFuncSetAttribute(k_graph_cg<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStageMax) != cudaSuccess ||
      cudaFuncSetAttribute(k_graph_cg<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStageMax) != cudaSuccess) {
    delete h;
    return gfail(BX_ECUDA, "bx_graph_create: shared memory attribute");
  }
  const size_t big = (size_t)n * max_rhs;
  bool ok = true;
  for (int l = 0; l <= h->lc[1] && ok; ++l) {
    const bx_graph_level& src = levels[l];
    Level L;
    L.n = src.n;
    L.nnz = src.nnz;
    L.ptr = h->alloc<int>(src.n + 1);
    L.col = h->alloc<int>(src.nnz);
    L.val = h->alloc<double>(src.nnz);
    L.dinv = h->alloc<double>(src.n);
    L.x = h->alloc<double>((size_t)src.n * max_rhs);
    L.s = h->alloc<double>((size_t)src.n * max_rhs);
    if (l > 0) L.b = h->alloc<double>((size_t)src.n * max_rhs);
    ok = L.ptr && L.col && L.val && L.dinv && L.x && L.s && (l == 0 || L.b);
    if (!ok) break;
    std::vector<double> dinv(src.n, 0.0);
    for (int i = 0; i < src.n; ++i)
      for (int p = src.row_ptr[i]; p < src.row_ptr[i + 1]; ++p)
        if (src.col[p] == i && src.val[p] != 0.0) dinv[i] = 1.0 / src.val[p];
    ok = cudaMemcpy(L.ptr, src.row_ptr, (size_t)(src.n + 1) * 4, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(L.col, src.col, (size_t)src.nnz * 4, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(L.val, src.val, (size_t)src.nnz * 8, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(L.dinv, dinv.data(), (size_t)src.n * 8, cudaMemcpyHostToDevice) == cudaSuccess;
    h->lv.push_back(L);
  }
  if (ok) {
    h->w_ptr = h->alloc<int>(n + 1);
    h->w_col = h->alloc<int>(weighted->nnz);
    h->w_val = h->alloc<double>(weighted->nnz);
    h->area = h->alloc<double>(n);
    for (double** v : {&h->R, &h->Z, &h->P0, &h->P1, &h->Q, &h->T1, &h->T2}) *v = h->alloc<double>(big);
    h->part = h->alloc<double>((size_t)2 * 3 * h->grid * max_rhs);
    h->scal = h->alloc<double>((size_t)8 * h->grid * max_rhs);
    h->out = h->alloc<double>(4 + 8);      // and the column groups' residuals
    h->ctl = h->alloc<unsigned>(4);
    ok = h->w_ptr && h->w_col && h->w_val && h->area && h->R && h->Z && h->P0 && h->P1 && h->Q && h->T1 && h->T2 &&
         h->part && h->scal && h->out && h->ctl;
    ok = ok && cudaMemcpy(h->w_ptr, weighted->row_ptr, (size_t)(n + 1) * 4, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(h->w_col, weighted->col, (size_t)weighted->nnz * 4, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(h->w_val, weighted->val, (size_t)weighted->nnz * 8, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(h->area, vor_sa, (size_t)n * 8, cudaMemcpyHostToDevice) == cudaSuccess;
  }
  if (!ok) {
    cudaGetLastError();
    delete h;
    return gfail(BX_ENOMEM, "bx_graph_create: device allocation or upload failed");
  }
  for (int l : h->lc) {
    Level& D = h->lv[l];
    if (D.dense) continue;
    if (l == n_levels - 1) {               // the coarsest: the caller's pseudo-inverse
      D.dense = h->alloc<double>((size_t)D.n * D.n);
      if (!D.dense || cudaMemcpy(D.dense, coarse_pinv, (size_t)D.n * D.n * 8, cudaMemcpyHostToDevice) != cudaSuccess)
        rc = gfail(BX_ENOMEM, "bx_graph_create: coarsest level");
    } else {
      rc = build_pinv(h, D, levels[l]);
    }
    if (rc != BX_OK) {
      cudaGetLastError();
      delete h;
      return rc;
    }
  }
  *out = h;
  return BX_OK;
}

extern "C" int bx_graph_solve(bx_graph_handle h, const double* B, double* X, int nrhs, double tol, int max_iter,
                              int* iters, double* rel_res, void* stream) {
  if (!h || !B || !X || nrhs < 1 || nrhs > h->max_rhs || max_iter < 1)
    return gfail(BX_EINVAL, "bx_graph_solve: bad arguments (nrhs must be 1..max_rhs)");
  return solve(h, B, X, nrhs, tol, max_iter, iters, rel_res, static_cast<cudaStream_t>(stream));
}

extern "C" int bx_lap_gj_apply(bx_graph_handle h, const double* X, double* Y, int nrhs, double tol, int max_iter,
                               int* iters, double* rel_res, void* stream) {
  if (!h || !X || !Y || nrhs < 1 || nrhs > h->max_rhs || max_iter < 1)
    return gfail(BX_EINVAL, "bx_lap_gj_apply: bad arguments (nrhs must be 1..max_rhs)");
  return lap_gj(h, X, Y, nrhs, tol, max_iter, iters, rel_res, static_cast<cudaStream_t>(stream));
}

extern "C" int bx_lap_gj_dense(bx_graph_handle h, double tol, int max_iter, int* iters, double* rel_res,
                               void* stream, bx_dense_op_handle* out) {
  if (!h || !out || max_iter < 1) return gfail(BX_EINVAL, "bx_lap_gj_dense: bad arguments");
  *out = nullptr;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  bx_dense_op_handle op = nullptr;
  int rc = bx_dense_op_create_empty(h->n, &op);
  if (rc != BX_OK) return rc;
  // blocks of whole 64-column tiles
  const int K = std::max(64, h->max_rhs / 64 * 64);
  if (K > h->max_rhs) {
    bx_dense_op_destroy(op);
    return gfail(BX_EINVAL, "bx_lap_gj_dense: the solver needs max_rhs >= 64");
  }
  double* Y = nullptr;
  if (cudaMalloc(&Y, (size_t)h->n * K * sizeof(double)) != cudaSuccess) {
    cudaGetLastError();
    bx_dense_op_destroy(op);
    return gfail(BX_ENOMEM, "bx_lap_gj_dense: column block");
  }
  int worst_it = 0;
  double worst_res = 0.0;
  for (int c0 = 0; c0 < h->n && rc == BX_OK; c0 += K) {
    const int k = std::min(K, h->n - c0);
    int it = 0;
    double res = 0.0;
    rc = lap_gj(h, nullptr, Y, k, tol, max_iter, &it, &res, s, true, c0);
    if (rc == BX_OK) rc = bx_dense_op_set_columns(op, c0, k, Y, s);
    worst_it = std::max(worst_it, it);
    worst_res = std::max(worst_res, res);
  }
  if (rc == BX_OK && cudaStreamSynchronize(s) != cudaSuccess) rc = gfail(BX_ECUDA, "bx_lap_gj_dense: build failed");
  cudaFree(Y);
  if (rc != BX_OK) {
    bx_dense_op_destroy(op);
    return rc;
  }
  if (iters) *iters = worst_it;
  if (rel_res) *rel_res = worst_res;
  *out = op;
  return BX_OK;
}

extern "C" int bx_graph_barrier_check(bx_graph_handle h, int* timed_out) {
  if (!h || !timed_out) return gfail(BX_EINVAL, "null argument");
  constexpr int kStuck = 0x80;             // a count that no wait can reach
  GCK(cudaMemset(h->T1, 0, (size_t)h->n * sizeof(double)));
  int rc = solve_async(h, h->T1, h->T2, 1, 1e-12, 4, 0, nullptr, kStuck);
  if (rc != BX_OK) return rc;
  *timed_out = solve_result(h, 1, nullptr, nullptr, nullptr) == BX_ECUDA ? 1 : 0;
  // the dense level's inverse: one node, in the workspace (each array two doubles at least)
  GCK(cudaMemset(h->Q, 0, sizeof(double)));
  GCK(cudaMemset(h->P0, 0, sizeof(int)));
  rc = run_pinv(PinvArgs{1, h->T1, h->T2, reinterpret_cast<const int*>(h->P0), h->Q, h->ctl}, 1, kStuck);
  *timed_out = *timed_out && rc == BX_ECUDA ? 1 : 0;
  GCK(cudaGetLastError());
  return BX_OK;
}

extern "C" int bx_graph_destroy(bx_graph_handle h) {
  delete h;
  return BX_OK;
}
