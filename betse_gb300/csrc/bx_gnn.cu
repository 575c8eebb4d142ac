// bx_gnn.cu -- the warm-start graph network: training and inference kernels.
//
// A 3-layer message-passing network on the cell adjacency (cells.cell_nn,
// betse/science/cells.py:1498-1533) predicts each cell's steady-state ion
// concentrations and Vmem from its channel diffusivities, pump rate and
// gap-junction conductance; the time stepping then runs from that prediction
// until its own residual test (max |dVm/dt|, sim.py:2083) passes.  BETSE has
// no counterpart: its init phase always starts from the uniform profile.
//
// Every layer is 64 wide (inputs zero-padded, the first n_out outputs used):
//   H0 = relu(X W0^T + b0)
//   A_l = mean over neighbours of H_{l-1}
//   R_l = relu(H_{l-1} Ws_l^T + A_l Wn_l^T + b_l),  H_l = H_{l-1} + R_l   (l = 1..3)
//   Yhat = H3 Wd^T + bd
// Training is BF16 with FP32 master weights: products read BF16 copies of the
// weights and BF16 activations and accumulate in FP32; gradients and Adam
// moments are FP32.  A forward layer is a tall product [nodes x 64] [64 x 64]
// (two of them for a message layer): it runs on the tensor cores, one CTA per
// 128 nodes, the activation tile and the weights staged in shared memory in
// the canonical K-major core-matrix layout, tcgen05.mma (BF16 x BF16 -> FP32
// in TMEM, M = 128, N = 64, K = 16 per instruction) issued by one thread, and
// four warps reading the accumulator back for the bias, activation and
// residual epilogue.  The backward takes FP32 gradients and stays on the
// FMA pipe: one kernel per layer, both products from one tile in shared
// memory.  Weight gradients are per-CTA partial sums, added in a fixed order
// by the kernel that applies Adam.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/bx.h"
#include "bx_tc.cuh"

// error text for bx_last_error (defined with the other entry points)
void bx_record_error(const char* msg);

namespace bxn {

using bf16 = __nv_bfloat16;
constexpr int W = 64, NMP = 3;
constexpr int OFF_W0 = 0, OFF_B0 = W * W, OFF_MP = OFF_B0 + W, MP_STRIDE = 2 * W * W + W;
constexpr int OFF_WD = OFF_MP + NMP * MP_STRIDE, OFF_BD = OFF_WD + W * W, NP = OFF_BD + W;
constexpr int kThreads = 256;
constexpr unsigned FULL = 0xffffffffu;

// activation planes, each [rows][W] BF16
enum Plane { P_X = 0, P_H0, P_H1, P_H2, P_H3, P_A1, P_A2, P_A3, P_R1, P_R2, P_R3, N_PLANES };

__device__ __forceinline__ float2 ld_bf2(const bf16* row, int lane) {
  return __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(row)[lane]);
}

// Programmatic dependent launch: every kernel of a pass waits for the one
// before it here, after it has fetched what no kernel of the pass writes (the
// weights, the graph), and lets the next one start as it ends.
__device__ __forceinline__ void grid_wait() {
#if defined(__CUDA_ARCH__) && (__CUDA_ARCH__ >= 900)
  cudaGridDependencySynchronize();
#endif
}

// ---- forward layers on the tensor cores
constexpr int kTcRows = 128;                         // nodes per CTA (the MMA's M)
constexpr int kTcThreads = 256;                      // warp w: TMEM lanes 32 (w % 4) ..., half of the columns
constexpr int kActTile = kTcRows * W * 2;            // 16 KB of BF16
constexpr int kWTile = W * W * 2;                    // 8 KB
constexpr int kTcSmem = 2 * (kActTile + kWTile) + 1024;   // two inputs (MODE 1)
constexpr int kTcSmem1 = kActTile + kWTile + 1024;        // one input (MODE 0, 2)
// kind::f16: FP32 accumulator, BF16 A and B, both K-major, N = 64, M = 128
constexpr uint32_t kIdescFwd = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(W >> 3) << 17) |
                               ((uint32_t)(kTcRows >> 4) << 24);

// A tile of ROWS rows of a row-major [*][64] BF16 array is ROWS * 8 pieces of
// 16 bytes; thread t holds pieces t, t + 256, ...  All of a thread's loads
// are issued before any store, so a tile costs one memory round trip.
template <int ROWS>
__device__ __forceinline__ void load_rows(uint4 (&v)[ROWS * 8 / kTcThreads], const bf16* __restrict__ src,
                                          int valid) {
  static_assert(ROWS * 8 % kTcThreads == 0, "whole pieces per thread");
#pragma unroll
  for (int j = 0; j < ROWS * 8 / kTcThreads; ++j) {
    const int e = (int)threadIdx.x + j * kTcThreads, r = e >> 3, c = e & 7;
    v[j] = r < valid ? reinterpret_cast<const uint4*>(src + (size_t)r * W)[c] : make_uint4(0u, 0u, 0u, 0u);
  }
}

// The pieces into the canonical no-swizzle K-major layout: 8 x 16-byte core
// matrices, the 8 K-adjacent cores of an 8-row group contiguous (128 B
// apart), 8-row groups 1024 B apart; rows at or past `valid` are zero.
template <int ROWS>
__device__ __forceinline__ void store_rows(uint8_t* tile, const uint4 (&v)[ROWS * 8 / kTcThreads]) {
#pragma unroll
  for (int j = 0; j < ROWS * 8 / kTcThreads; ++j) {
    const int e = (int)threadIdx.x + j * kTcThreads, r = e >> 3, c = e & 7;
    *reinterpret_cast<uint4*>(tile + ((r >> 3) * 8 + c) * 128 + (r & 7) * 16) = v[j];
  }
}

// eight FP32 values to 16 bytes of BF16
__device__ __forceinline__ uint4 pack_bf8(const float (&v)[8]) {
  uint4 u;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int q = 0; q < 4; ++q) h[q] = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
  return u;
}

struct FwdArgs {
  int n;
  const bf16* in1;                 // [n][W]; MODE 0 writes it (the padded inputs)
  bf16* in2;                       // MODE 1: the neighbour means, written here
  const bf16* wb;
  int off_w1, off_w2;
  const float* master;
  int off_b;
  bf16 *outR, *outH;
  float* outY;
  int n_out;
  unsigned* err;
  const float* x;                  // MODE 0: [n][n_in]
  int n_in;
  const int *ptr, *nbr;            // MODE 1: adjacency
  int lo;
};

// MODE 0: encoder  H = relu(x W1^T + b), x zero-padded to W columns in BF16
// MODE 1: message  R = relu(in1 W1^T + A W2^T + b), H = in1 + R, A the mean of
//                  in1 over the neighbours: gathered eight lanes a node
//                  (16 bytes each), four rows in flight, summed in list order
// MODE 2: decoder  Y = in1 W1^T + b (FP32, first n_out columns)
// Bound by latency (gather, tile, MMA, read-back in sequence): with the inputs
// packed and the means formed by kernels of their own a forward pass of 30,858
// nodes took 92 us, 85 now (and four launches fewer).
// A wait that runs out (about two seconds) raises *err and leaves the rows
// unwritten; the TMEM is freed either way.
template <int MODE>
__global__ void __launch_bounds__(kTcThreads) k_fwd_tc(FwdArgs a) {
  const int n = a.n, n_out = a.n_out;
  const bf16 *in1 = a.in1, *wb = a.wb;
  const float* master = a.master;
  const int off_w1 = a.off_w1, off_w2 = a.off_w2, off_b = a.off_b;
  bf16 *outR = a.outR, *outH = a.outH;
  float* outY = a.outY;
  unsigned* err = a.err;
  using namespace bxtc;
  extern __shared__ uint8_t tc_smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* a1 = sm;
  uint8_t* b1 = a1 + kActTile;
  uint8_t* a2 = b1 + kWTile;
  uint8_t* b2 = a2 + kActTile;
  __shared__ __align__(8) uint64_t done;
  __shared__ uint32_t tmem_base;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r0 = blockIdx.x * kTcRows;
  const int valid = min(kTcRows, n - r0);

  {
    uint4 w1[W * 8 / kTcThreads], w2[W * 8 / kTcThreads];
    load_rows<W>(w1, wb + off_w1, W);
    if (MODE == 1) load_rows<W>(w2, wb + off_w2, W);
    store_rows<W>(b1, w1);
    if (MODE == 1) store_rows<W>(b2, w2);
  }
  if (MODE == 0) {
    grid_wait();
    for (int e = (int)threadIdx.x; e < kTcRows * 8; e += kTcThreads) {
      const int r = e >> 3, c = e & 7;
      float v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        v[q] = r < valid && 8 * c + q < a.n_in ? a.x[(size_t)(r0 + r) * a.n_in + 8 * c + q] : 0.f;
      const uint4 u = pack_bf8(v);
      if (r < valid) reinterpret_cast<uint4*>(const_cast<bf16*>(in1) + (size_t)(r0 + r) * W)[c] = u;
      *reinterpret_cast<uint4*>(a1 + ((r >> 3) * 8 + c) * 128 + (r & 7) * 16) = u;
    }
  } else if (MODE == 1) {
    constexpr int NP8 = kTcThreads / 8, NIT = kTcRows / NP8;      // nodes a pass, passes
    const int g8 = (int)threadIdx.x >> 3, c = (int)threadIdx.x & 7;
    int pa[NIT], pb[NIT], nb[NIT];
#pragma unroll
    for (int it = 0; it < NIT; ++it) {
      const int r = g8 + it * NP8;
      pa[it] = r < valid ? a.ptr[a.lo + r0 + r] : 0;
      pb[it] = r < valid ? a.ptr[a.lo + r0 + r + 1] : 0;
    }
#pragma unroll
    for (int it = 0; it < NIT; ++it) nb[it] = pa[it] + c < pb[it] ? a.nbr[pa[it] + c] : -1;
    grid_wait();
    uint4 va[kTcRows * 8 / kTcThreads];
    load_rows<kTcRows>(va, in1 + (size_t)r0 * W, valid);
#pragma unroll
    for (int it = 0; it < NIT; ++it) {
      const int r = g8 + it * NP8, deg = pb[it] - pa[it];
      int most = deg;
#pragma unroll
      for (int o = 8; o < 32; o <<= 1) most = max(most, __shfl_xor_sync(FULL, most, o));
      float s[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) s[q] = 0.f;
      for (int p0 = 0; p0 < most; p0 += 8) {
        if (p0 > 0) nb[it] = pa[it] + p0 + c < pb[it] ? a.nbr[pa[it] + p0 + c] : -1;
#pragma unroll
        for (int k0 = 0; k0 < 8; k0 += 4) {
          if (p0 + k0 >= most) break;
          uint4 h[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int j = __shfl_sync(FULL, nb[it], k0 + u, 8);
            h[u] = j >= 0 ? reinterpret_cast<const uint4*>(in1 + (size_t)(j - a.lo) * W)[c] : make_uint4(0u, 0u, 0u, 0u);
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const __nv_bfloat162* b2v = reinterpret_cast<const __nv_bfloat162*>(&h[u]);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const float2 f = __bfloat1622float2(b2v[q]);
              s[2 * q] += f.x;
              s[2 * q + 1] += f.y;
            }
          }
        }
      }
      if (deg > 0)
#pragma unroll
        for (int q = 0; q < 8; ++q) s[q] /= (float)deg;
      const uint4 u = pack_bf8(s);
      if (r < valid) reinterpret_cast<uint4*>(a.in2 + (size_t)(r0 + r) * W)[c] = u;
      *reinterpret_cast<uint4*>(a2 + ((r >> 3) * 8 + c) * 128 + (r & 7) * 16) = u;
    }
    store_rows<kTcRows>(a1, va);
  } else {
    grid_wait();
    uint4 va[kTcRows * 8 / kTcThreads];
    load_rows<kTcRows>(va, in1 + (size_t)r0 * W, valid);
    store_rows<kTcRows>(a1, va);
  }
  // the tensor core reads shared memory through the async proxy
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&done), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(W));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base;

  if (threadIdx.x == 0) {
#pragma unroll
    for (int kk = 0; kk < W / 16; ++kk) {     // two K-adjacent core matrices per MMA (K = 16)
      const uint32_t o = (uint32_t)kk * 256u;
      mma_f16(tmem, smem_desc(smem_u32(a1) + o, 128, 1024), smem_desc(smem_u32(b1) + o, 128, 1024), kIdescFwd,
              kk > 0 ? 1u : 0u);
    }
    if (MODE == 1)
#pragma unroll
      for (int kk = 0; kk < W / 16; ++kk) {
        const uint32_t o = (uint32_t)kk * 256u;
        mma_f16(tmem, smem_desc(smem_u32(a2) + o, 128, 1024), smem_desc(smem_u32(b2) + o, 128, 1024), kIdescFwd,
                1u);
      }
    mma_commit(smem_u32(&done));
  }
  __syncwarp();
  const bool ok = __all_sync(FULL, mbar_wait(smem_u32(&done), 0u));
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (ok) {
    constexpr int HC = W / 2;                        // this warp's columns
    const int f0 = (warp >> 2) * HC, r = r0 + (warp & 3) * 32 + lane;
    float v[HC];
#pragma unroll
    for (int c0 = 0; c0 < HC; c0 += 16)
      tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(f0 + c0), v + c0);
    if (r < n) {
      const size_t o = (size_t)r * W + f0;
#pragma unroll
      for (int f = 0; f < HC; ++f) v[f] += master[off_b + f0 + f];
      if (MODE == 2) {
#pragma unroll
        for (int f = 0; f < HC; ++f)          // constant indices keep v in registers
          if (f0 + f < n_out) outY[(size_t)r * n_out + f0 + f] = v[f];
      } else {
#pragma unroll
        for (int f8 = 0; f8 < HC; f8 += 8) {
          __align__(16) bf16 rr[8], hh[8];
          uint4 x = make_uint4(0u, 0u, 0u, 0u);
          if (MODE == 1) x = reinterpret_cast<const uint4*>(in1 + o)[f8 / 8];
          const bf16* xb = reinterpret_cast<const bf16*>(&x);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            rr[q] = __float2bfloat16_rn(fmaxf(v[f8 + q], 0.f));
            hh[q] = MODE == 1 ? __float2bfloat16_rn(__bfloat162float(xb[q]) + __bfloat162float(rr[q])) : rr[q];
          }
          if (MODE == 1) reinterpret_cast<uint4*>(outR + o)[f8 / 8] = *reinterpret_cast<const uint4*>(rr);
          reinterpret_cast<uint4*>(outH + o)[f8 / 8] = *reinterpret_cast<const uint4*>(hh);
        }
      }
    }
  } else if (lane == 0) {
    atomicOr(err, 1u);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(W));
  }
}

// ---- backward: one kernel per layer
// A layer's backward is two FP32 products with the same left factor dZ: the
// input gradients dZ [W1 | W2] (over the layer's outputs) and the weight
// gradients dZ^T [In1 | In2] (over the nodes).  Both run from one shared copy
// of the tile in register tiles of 8 x 4 per thread (three 16-byte shared
// reads per 32 FMA); the weight gradients stay in registers over all of a
// CTA's rows.  dIn is formed while the tile is loaded: the residual path plus
// the transposed neighbour mean of the layer above's G.  Bound by the FMA pipe
// (the gradients are FP32); with a warp per node, operands by shuffle and the
// weight gradients in their own passes a training step of 30,858 nodes took
// 680 us, its call included, 270 now (a middle layer 109 us before, 38 to 44 now).
constexpr int kBwdT = 256, kBwdRows = 64, kBwdPerSM = 2;

struct BwdArgs {
  int n, lo, per;                          // nodes, first node of the range, rows per CTA
  const float* dH;                         // residual path [n][W]
  const float* G;                          // layer above: dZ W2, null at the top
  const int *ptrT, *nbrT;
  const float* inv_deg;
  const bf16 *mask, *in1, *in2;
  const bf16* wb;
  int off_w1, off_w2;
  float *outH, *outG;
  float* part;                             // [grid][NP]
  int off_part;
  const float *yhat, *y;                   // TOP
  int n_out;
  float* loss_part;
};

enum BwdMode { BWD_TOP = 0, BWD_MID = 1, BWD_ENC = 2 };
template <int MODE>
struct BwdShape {
  static constexpr int cols = MODE == BWD_MID ? 2 * W : W;      // of [W1 | W2] and [In1 | In2]
  static constexpr int smem = 4 * ((MODE == BWD_ENC ? 0 : W * cols) + kBwdRows * cols + kBwdRows * W +
                                   (MODE == BWD_MID ? kBwdRows * W : 0));
};

template <int N>
__device__ __forceinline__ void ld_vec(float (&v)[N], const float* p) {
  if (N == 4) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x; v[1] = q.y; v[2 % N] = q.z; v[3 % N] = q.w;
  } else {
    const float2 q = *reinterpret_cast<const float2*>(p);
    v[0] = q.x; v[1] = q.y;
  }
}
template <int N>
__device__ __forceinline__ void st_vec(float* p, const float (&v)[N]) {
  if (N == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2 % N], v[3 % N]);
  else *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
}

// TOP: dZ = dY = 2 (Yhat - Y) / (N n_out), loss; dH = dZ Wd; dWd, dbd
// MID: dIn = dH + aggT(G), dZ = dIn * (R > 0); dH' = dIn + dZ W1, G' = dZ W2; dW1, dW2, db
// ENC: dIn likewise, dZ = dIn * (H0 > 0); dW0, db0
template <int MODE>
__global__ void __launch_bounds__(kBwdT, kBwdPerSM) k_bwd(BwdArgs a) {
  constexpr int NCOL = BwdShape<MODE>::cols, CPT = NCOL / 32;
  extern __shared__ float bs[];
  float* sIn = bs;
  float* sZ = sIn + kBwdRows * NCOL;
  float* sD = sZ + kBwdRows * W;                                 // MID
  float* sW = sD + (MODE == BWD_MID ? kBwdRows * W : 0);         // TOP, MID
  __shared__ float red[kBwdT / 32];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int row0 = blockIdx.x * a.per, row1 = min(a.n, row0 + a.per);
  const int nchunk = (a.per + kBwdRows - 1) / kBwdRows;
  const int chunk = ((a.per + nchunk - 1) / nchunk + 7) & ~7;     // even chunks, whole groups of eight

  if (MODE != BWD_ENC) {
    for (int e = t; e < W * W / 2; e += kBwdT) {
      const int f = 2 * e / W, c = 2 * e - f * W;
      const float2 w1 = ld_bf2(a.wb + a.off_w1, e);
      sW[f * NCOL + c] = w1.x;
      sW[f * NCOL + c + 1] = w1.y;
      if (MODE == BWD_MID) {
        const float2 w2 = ld_bf2(a.wb + a.off_w2, e);
        sW[f * NCOL + W + c] = w2.x;
        sW[f * NCOL + W + c + 1] = w2.y;
      }
    }
  }
  grid_wait();
  const int F = MODE == BWD_TOP ? a.n_out : W;                   // rows of dZ^T that are not zero
  const float scale = MODE == BWD_TOP ? 2.0f / ((float)a.n * (float)a.n_out) : 0.f;
  float acc[8][CPT], bacc = 0.f, loss = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int c = 0; c < CPT; ++c) acc[j][c] = 0.f;

  for (int i0 = row0; i0 < row1; i0 += chunk) {
    const int rows = min(chunk, row1 - i0);
    __syncthreads();                                             // the tile of the chunk before is done with
    // ---- the layer's inputs
#pragma unroll 4
    for (int q = t; q < rows * (NCOL / 8); q += kBwdT) {
      const int r = q / (NCOL / 8), c8 = q - r * (NCOL / 8);
      const bf16* src = (MODE == BWD_MID && c8 >= W / 8 ? a.in2 : a.in1) + (size_t)(i0 + r) * W + (c8 & 7) * 8;
      const uint4 v = *reinterpret_cast<const uint4*>(src);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
      const float2 f0 = __bfloat1622float2(h[0]), f1 = __bfloat1622float2(h[1]);
      const float2 f2 = __bfloat1622float2(h[2]), f3 = __bfloat1622float2(h[3]);
      float4* d = reinterpret_cast<float4*>(sIn + r * NCOL + c8 * 8);
      d[0] = make_float4(f0.x, f0.y, f1.x, f1.y);
      d[1] = make_float4(f2.x, f2.y, f3.x, f3.y);
    }
    // ---- dZ
    if (MODE == BWD_TOP) {
      for (int q = t; q < rows * (W / 4); q += kBwdT)
        reinterpret_cast<float4*>(sZ)[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      __syncthreads();
#pragma unroll 4
      for (int q = t; q < rows * a.n_out; q += kBwdT) {
        const int r = q / a.n_out, f = q - r * a.n_out;
        const size_t o = (size_t)i0 * a.n_out + q;
        const float e = a.yhat[o] - a.y[o];
        loss += e * e;
        sZ[r * W + f] = scale * e;
      }
    } else {
      // half a warp per node, four features a lane
      const int hw = t >> 4, l16 = t & 15;
      constexpr int NH = kBwdT / 16, NIT = kBwdRows / NH;
      int pa[NIT], pb[NIT];
#pragma unroll
      for (int it = 0; it < NIT; ++it) {
        const int r = hw + it * NH;
        const bool in = a.G && r < rows;
        pa[it] = in ? a.ptrT[a.lo + i0 + r] : 0;
        pb[it] = in ? a.ptrT[a.lo + i0 + r + 1] : 0;
      }
      int nb[NIT];
      float wt[NIT];
#pragma unroll
      for (int it = 0; it < NIT; ++it) {
        const int p = pa[it] + l16;
        nb[it] = p < pb[it] ? a.nbrT[p] : -1;
      }
#pragma unroll
      for (int it = 0; it < NIT; ++it) wt[it] = nb[it] >= 0 ? a.inv_deg[nb[it]] : 0.f;
#pragma unroll
      for (int it0 = 0; it0 < NIT; it0 += 2) {               // two nodes a half-warp: eight rows in flight
        float4 s[2], d[2];
        uint2 mk[2];
        int most = 0;
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          const int r = hw + (it0 + v) * NH;
          s[v] = d[v] = make_float4(0.f, 0.f, 0.f, 0.f);
          mk[v] = make_uint2(0u, 0u);
          if (r < rows) {
            d[v] = reinterpret_cast<const float4*>(a.dH + (size_t)(i0 + r) * W)[l16];
            mk[v] = reinterpret_cast<const uint2*>(a.mask + (size_t)(i0 + r) * W)[l16];
          }
          most = max(most, pb[it0 + v] - pa[it0 + v]);
        }
        most = max(most, __shfl_xor_sync(FULL, most, 16));
        for (int p0 = 0; p0 < most; p0 += 16) {
          if (p0 > 0) {
#pragma unroll
            for (int v = 0; v < 2; ++v) {
              const int p = pa[it0 + v] + p0 + l16;
              nb[it0 + v] = p < pb[it0 + v] ? a.nbrT[p] : -1;
              wt[it0 + v] = nb[it0 + v] >= 0 ? a.inv_deg[nb[it0 + v]] : 0.f;
            }
          }
          for (int k0 = 0; k0 < min(16, most - p0); k0 += 4) {
            float4 g[2][4];
#pragma unroll
            for (int v = 0; v < 2; ++v)
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const int i = __shfl_sync(FULL, nb[it0 + v], k0 + u, 16);
                g[v][u] = i >= 0 ? reinterpret_cast<const float4*>(a.G + (size_t)(i - a.lo) * W)[l16]
                                 : make_float4(0.f, 0.f, 0.f, 0.f);
              }
#pragma unroll
            for (int v = 0; v < 2; ++v)
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const float w = __shfl_sync(FULL, wt[it0 + v], k0 + u, 16);
                s[v].x = fmaf(g[v][u].x, w, s[v].x);
                s[v].y = fmaf(g[v][u].y, w, s[v].y);
                s[v].z = fmaf(g[v][u].z, w, s[v].z);
                s[v].w = fmaf(g[v][u].w, w, s[v].w);
              }
          }
        }
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          const int r = hw + (it0 + v) * NH;
          if (r >= rows) continue;
          float4 x = d[v];
          x.x += s[v].x; x.y += s[v].y; x.z += s[v].z; x.w += s[v].w;
          if (MODE == BWD_MID) *reinterpret_cast<float4*>(sD + r * W + 4 * l16) = x;
          const float2 m0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&mk[v].x));
          const float2 m1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&mk[v].y));
          if (!(m0.x > 0.f)) x.x = 0.f;
          if (!(m0.y > 0.f)) x.y = 0.f;
          if (!(m1.x > 0.f)) x.z = 0.f;
          if (!(m1.y > 0.f)) x.w = 0.f;
          *reinterpret_cast<float4*>(sZ + r * W + 4 * l16) = x;
        }
      }
    }
    __syncthreads();
    // ---- input gradients: warp = 8 nodes, lane = CPT columns
    if (MODE != BWD_ENC && warp * 8 < rows) {
      float o[8][CPT];
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int c = 0; c < CPT; ++c) o[j][c] = 0.f;
      const float* z0 = sZ + warp * 8 * W;                       // (rows past the last are read, not used)
#pragma unroll 2
      for (int f = 0; f < F; f += 4) {
        float z[8][4];
#pragma unroll
        for (int j = 0; j < 8; ++j) ld_vec<4>(z[j], z0 + j * W + f);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float w[CPT];
          ld_vec<CPT>(w, sW + (f + q) * NCOL + lane * CPT);
#pragma unroll
          for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int c = 0; c < CPT; ++c) o[j][c] = fmaf(z[j][q], w[c], o[j][c]);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int r = warp * 8 + j;
        if (r >= rows) break;
        const size_t g = (size_t)(i0 + r) * W;
        if (MODE == BWD_TOP) {
          st_vec<CPT>(a.outH + g + lane * CPT, o[j]);
        } else if (lane < 16) {
          const float4 d = *reinterpret_cast<const float4*>(sD + r * W + 4 * lane);
          o[j][0] = d.x + o[j][0];
          o[j][1] = d.y + o[j][1];
          o[j][2 % CPT] = d.z + o[j][2 % CPT];
          o[j][3 % CPT] = d.w + o[j][3 % CPT];
          st_vec<CPT>(a.outH + g + 4 * lane, o[j]);
        } else {
          st_vec<CPT>(a.outG + g + 4 * (lane - 16), o[j]);
        }
      }
    }
    // ---- weight gradients: warp = 8 rows of dZ^T, lane = CPT columns
    if (warp * 8 < F) {
#pragma unroll 4
      for (int r = 0; r < rows; ++r) {
        float z[2][4], x[CPT];
        ld_vec<4>(z[0], sZ + r * W + warp * 8);
        ld_vec<4>(z[1], sZ + r * W + warp * 8 + 4);
        ld_vec<CPT>(x, sIn + r * NCOL + lane * CPT);
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int c = 0; c < CPT; ++c) acc[j][c] = fmaf(z[j >> 2][j & 3], x[c], acc[j][c]);
      }
    }
    for (int r = t >> 6; r < rows; r += kBwdT / W) bacc += sZ[r * W + (t & (W - 1))];
  }
  __syncthreads();
  float* pb = a.part + (size_t)blockIdx.x * NP + a.off_part;
  if (warp * 8 < F) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int f = warp * 8 + j, c = lane * CPT;
      st_vec<CPT>(pb + (c >= W ? W * W + c - W : c) + f * W, acc[j]);
    }
  }
  sZ[t] = bacc;
  if (MODE == BWD_TOP) {
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(FULL, loss, o);
    if (lane == 0) red[warp] = loss;
  }
  __syncthreads();
  if (t < W) pb[W * NCOL + t] = ((sZ[t] + sZ[t + W]) + sZ[t + 2 * W]) + sZ[t + 3 * W];
  if (MODE == BWD_TOP && t == 0) {
    float s = 0.f;
    for (int w = 0; w < kBwdT / 32; ++w) s += red[w];
    a.loss_part[blockIdx.x] = s;
  }
}

// The CTAs' partials of every gradient (32 parameters a block, eight threads
// each, added in a fixed order), then Adam's update of the parameter; the last
// block adds the loss.  Latency-bound: with one thread per parameter adding 304
// partials, layer by layer, this took 8 x 14.7 us, the loss 16.4 and Adam 4.3.
struct AdamArgs {
  float *master, *m, *v;
  bf16* wb;
  float lr, b1, b2, eps, bc1, bc2;
};
constexpr int kUpParams = 32, kUpSlices = 8;
template <bool ADAM>
__global__ void __launch_bounds__(kUpParams* kUpSlices) k_update(int nb, const float* __restrict__ part, int n_out,
                                                                const float* __restrict__ loss_part, float loss_scale,
                                                                float* __restrict__ loss, float* __restrict__ grad,
                                                                AdamArgs a) {
  __shared__ float red[kUpSlices][kUpParams];
  const int x = threadIdx.x % kUpParams, q = threadIdx.x / kUpParams;
  const bool last = blockIdx.x == gridDim.x - 1;
  const int e = blockIdx.x * kUpParams + x;
  float s = 0.f;
  if (last) {
    for (int b = threadIdx.x; b < nb; b += kUpParams * kUpSlices) s += loss_part[b];
  } else if (!(e >= OFF_WD && e < OFF_BD && (e - OFF_WD) / W >= n_out)) {   // (the decoder's unused rows: zero)
#pragma unroll 4
    for (int b = q; b < nb; b += kUpSlices) s += part[(size_t)b * NP + e];
  }
  red[q][x] = s;
  __syncthreads();
  if (q != 0) return;
  s = 0.f;
#pragma unroll
  for (int j = 0; j < kUpSlices; ++j) s += red[j][x];
  if (last) {
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
    if (x == 0) *loss = s * loss_scale;
    return;
  }
  if (!ADAM) {
    grad[e] = s;
    return;
  }
  const float mm = a.b1 * a.m[e] + (1.f - a.b1) * s;
  const float vv = a.b2 * a.v[e] + (1.f - a.b2) * s * s;
  a.m[e] = mm;
  a.v[e] = vv;
  const float w = a.master[e] - a.lr * (mm / a.bc1) / (sqrtf(vv / a.bc2) + a.eps);
  a.master[e] = w;
  a.wb[e] = __float2bfloat16_rn(w);
}
static_assert(NP % kUpParams == 0 && kUpParams == 32, "k_update: whole blocks, a warp of parameters");

__global__ void k_to_bf16(int np, const float* __restrict__ src, bf16* __restrict__ dst) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < np) dst[e] = __float2bfloat16_rn(src[e]);
}

}  // namespace bxn

struct bx_gnn {
  float *master = nullptr, *m = nullptr, *v = nullptr, *grad = nullptr;
  __nv_bfloat16* wb = nullptr;
  int n_graph = 0;
  int *ptr = nullptr, *nbr = nullptr, *ptrT = nullptr, *nbrT = nullptr;
  float* inv_deg = nullptr;
  int cap = 0;                              // activation rows
  __nv_bfloat16* act = nullptr;             // N_PLANES x [cap][W]
  float *yhat = nullptr, *dHa = nullptr, *dHb = nullptr, *Ga = nullptr, *Gb = nullptr;
  float *part = nullptr, *loss_part = nullptr;   // per backward CTA: every gradient, the loss
  float* loss = nullptr;                    // followed by err
  unsigned* err = nullptr;                  // a tensor-core wait ran out (k_fwd_tc)
  int step = 0;
  cudaStream_t stream = nullptr;
  std::vector<int> h_ptr, h_nbr;            // host copy: node ranges are checked for closure
  int ok_lo = -1, ok_hi = -1;               // last range found closed under adjacency
};

namespace {

using bxn::W;

int nfail(int code, const std::string& msg) {
  bx_record_error(msg.c_str());
  return code;
}
#define NX(call)                                                                            \
  do {                                                                                      \
    cudaError_t e_ = (call);                                                                \
    if (e_ != cudaSuccess) return nfail(BX_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

int ensure_cap(bx_gnn* h, int rows) {
  if (rows <= h->cap) return BX_OK;
  void* ptrs[] = {h->act, h->yhat, h->dHa, h->dHb, h->Ga, h->Gb};
  for (void* p : ptrs) cudaFree(p);
  h->act = nullptr;
  h->yhat = h->dHa = h->dHb = h->Ga = h->Gb = nullptr;
  h->cap = 0;
  const size_t r = (size_t)rows;
  if (cudaMalloc(&h->act, (size_t)bxn::N_PLANES * r * W * sizeof(__nv_bfloat16)) != cudaSuccess ||
      cudaMalloc(&h->yhat, r * W * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&h->dHa, r * W * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&h->dHb, r * W * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&h->Ga, r * W * sizeof(float)) != cudaSuccess ||
      cudaMalloc(&h->Gb, r * W * sizeof(float)) != cudaSuccess) {
    cudaGetLastError();
    return nfail(BX_ENOMEM, "cudaMalloc network activations");
  }
  h->cap = rows;
  return BX_OK;
}

__nv_bfloat16* plane(bx_gnn* h, int p) { return h->act + (size_t)p * h->cap * W; }

// after a synchronisation: did a tensor-core wait run out?
int check_tc(bx_gnn* h) {
  unsigned e = 0;
  NX(cudaMemcpy(&e, h->err, 4, cudaMemcpyDeviceToHost));
  if (e) return nfail(BX_ECUDA, "network: a tensor-core wait timed out");
  return BX_OK;
}

int check_range(bx_gnn* h, int lo, int hi) {
  if (!h->ptr) return nfail(BX_ESTATE, "network: bx_gnn_set_graph first");
  if (lo < 0 || hi <= lo || hi > h->n_graph) return nfail(BX_EINVAL, "network: node range outside the graph");
  if (lo != h->ok_lo || hi != h->ok_hi) {
    // every neighbour of a node in [lo, hi) must lie in [lo, hi) (whole clusters)
    for (int p = h->h_ptr[lo]; p < h->h_ptr[hi]; ++p)
      if (h->h_nbr[p] < lo || h->h_nbr[p] >= hi)
        return nfail(BX_EINVAL, "network: node range cuts through a cluster (neighbour outside the range)");
    h->ok_lo = lo;
    h->ok_hi = hi;
  }
  return ensure_cap(h, hi - lo);
}

template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kern)(KArgs...), unsigned grid, unsigned block, size_t smem, cudaStream_t s,
                       Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

int forward(bx_gnn* h, int lo, int hi, const float* x, int n_in, int n_out) {
  using namespace bxn;
  const int n = hi - lo;
  cudaStream_t s = h->stream;
  const unsigned g = (unsigned)((n + kTcRows - 1) / kTcRows);
  FwdArgs a{};
  a.n = n; a.wb = h->wb; a.master = h->master; a.err = h->err;
  a.x = x; a.n_in = n_in; a.ptr = h->ptr; a.nbr = h->nbr; a.lo = lo;
  a.in1 = plane(h, P_X); a.outH = plane(h, P_H0); a.off_w1 = OFF_W0; a.off_b = OFF_B0;
  // (an ordinary launch: the weights may come from the kernel before it)
  k_fwd_tc<0><<<g, kTcThreads, kTcSmem1, s>>>(a);
  for (int l = 0; l < NMP; ++l) {
    const int o = OFF_MP + l * MP_STRIDE;
    a.in1 = plane(h, P_H0 + l); a.in2 = plane(h, P_A1 + l); a.outR = plane(h, P_R1 + l); a.outH = plane(h, P_H1 + l);
    a.off_w1 = o; a.off_w2 = o + W * W; a.off_b = o + 2 * W * W;
    NX(launch_pdl(k_fwd_tc<1>, g, kTcThreads, kTcSmem, s, a));
  }
  a.in1 = plane(h, P_H3); a.outY = h->yhat; a.n_out = n_out; a.off_w1 = OFF_WD; a.off_b = OFF_BD;
  NX(launch_pdl(k_fwd_tc<2>, g, kTcThreads, kTcSmem1, s, a));
  NX(cudaGetLastError());
  return BX_OK;
}

constexpr int kBwdCtas = 152 * bxn::kBwdPerSM;
constexpr int kUpGrid = bxn::NP / bxn::kUpParams + 1, kUpThreads = bxn::kUpParams * bxn::kUpSlices;

// k_update then finishes the gradients; *nb: the CTAs whose partials it adds
int backward(bx_gnn* h, int lo, int hi, const float* y, int n_out, int* nb) {
  using namespace bxn;
  const int n = hi - lo;
  cudaStream_t s = h->stream;
  if (!h->part && cudaMalloc(&h->part, (size_t)kBwdCtas * NP * 4) != cudaSuccess) {
    cudaGetLastError();
    return nfail(BX_ENOMEM, "cudaMalloc network gradients");
  }
  BwdArgs a{};
  a.n = n; a.lo = lo;
  // one wave of two CTAs an SM, rows in whole groups of eight (a warp's)
  a.per = 8 * ((n + 8 * kBwdCtas - 1) / (8 * kBwdCtas));
  const unsigned g = (unsigned)((n + a.per - 1) / a.per);
  *nb = (int)g;
  a.ptrT = h->ptrT; a.nbrT = h->nbrT; a.inv_deg = h->inv_deg; a.wb = h->wb;
  a.part = h->part; a.loss_part = h->loss_part;
  a.yhat = h->yhat; a.y = y; a.n_out = n_out;
  a.in1 = plane(h, P_H3); a.off_w1 = OFF_WD; a.off_part = OFF_WD; a.outH = h->dHa;
  NX(launch_pdl(k_bwd<BWD_TOP>, g, kBwdT, BwdShape<BWD_TOP>::smem, s, a));
  float *dH = h->dHa, *dHn = h->dHb, *Gn = h->Ga, *Go = h->Gb;
  for (int l = NMP - 1; l >= 0; --l) {
    const int o = OFF_MP + l * MP_STRIDE;
    a.dH = dH; a.outH = dHn; a.outG = Gn;
    a.mask = plane(h, P_R1 + l); a.in1 = plane(h, P_H0 + l); a.in2 = plane(h, P_A1 + l);
    a.off_w1 = o; a.off_w2 = o + W * W; a.off_part = o;
    NX(launch_pdl(k_bwd<BWD_MID>, g, kBwdT, BwdShape<BWD_MID>::smem, s, a));
    a.G = Gn;
    std::swap(dH, dHn);
    std::swap(Gn, Go);
  }
  a.dH = dH; a.mask = plane(h, P_H0); a.in1 = plane(h, P_X); a.off_part = OFF_W0;
  NX(launch_pdl(k_bwd<BWD_ENC>, g, kBwdT, BwdShape<BWD_ENC>::smem, s, a));
  NX(cudaGetLastError());
  return BX_OK;
}

}  // namespace

extern "C" {

int bx_gnn_create(bx_gnn_handle* out) {
  if (!out) return nfail(BX_EINVAL, "null argument");
  bx_gnn* h = new bx_gnn();
  const size_t P = bxn::NP;
  if (cudaMalloc(&h->master, P * 4) != cudaSuccess || cudaMalloc(&h->m, P * 4) != cudaSuccess ||
      cudaMalloc(&h->v, P * 4) != cudaSuccess || cudaMalloc(&h->grad, P * 4) != cudaSuccess ||
      cudaMalloc(&h->wb, P * 2) != cudaSuccess ||
      cudaMalloc(&h->loss_part, (size_t)kBwdCtas * 4) != cudaSuccess || cudaMalloc(&h->loss, 8) != cudaSuccess ||
      cudaStreamCreate(&h->stream) != cudaSuccess) {
    cudaGetLastError();
    bx_gnn_destroy(h);
    return nfail(BX_ENOMEM, "cudaMalloc network parameters");
  }
  if (cudaFuncSetAttribute(bxn::k_fwd_tc<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, bxn::kTcSmem) !=
          cudaSuccess ||
      cudaFuncSetAttribute(bxn::k_fwd_tc<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, bxn::kTcSmem) !=
          cudaSuccess ||
      cudaFuncSetAttribute(bxn::k_fwd_tc<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, bxn::kTcSmem) !=
          cudaSuccess ||
      cudaFuncSetAttribute(bxn::k_bwd<bxn::BWD_TOP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           bxn::BwdShape<bxn::BWD_TOP>::smem) != cudaSuccess ||
      cudaFuncSetAttribute(bxn::k_bwd<bxn::BWD_MID>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           bxn::BwdShape<bxn::BWD_MID>::smem) != cudaSuccess) {
    cudaGetLastError();
    bx_gnn_destroy(h);
    return nfail(BX_ECUDA, "network: shared memory attribute of the layers");
  }
  h->err = reinterpret_cast<unsigned*>(h->loss + 1);
  cudaMemset(h->loss, 0, 8);
  cudaMemset(h->master, 0, P * 4);
  cudaMemset(h->m, 0, P * 4);
  cudaMemset(h->v, 0, P * 4);
  cudaMemset(h->wb, 0, P * 2);
  *out = h;
  return BX_OK;
}

int bx_gnn_n_params(void) { return bxn::NP; }

int bx_gnn_set_params(bx_gnn_handle h, const float* params) {
  if (!h || !params) return nfail(BX_EINVAL, "null argument");
  NX(cudaMemcpy(h->master, params, bxn::NP * 4, cudaMemcpyHostToDevice));
  NX(cudaMemset(h->m, 0, bxn::NP * 4));
  NX(cudaMemset(h->v, 0, bxn::NP * 4));
  bxn::k_to_bf16<<<(bxn::NP + 255) / 256, 256, 0, h->stream>>>(bxn::NP, h->master, h->wb);
  NX(cudaGetLastError());
  NX(cudaStreamSynchronize(h->stream));
  h->step = 0;
  return BX_OK;
}

int bx_gnn_get_params(bx_gnn_handle h, float* params) {
  if (!h || !params) return nfail(BX_EINVAL, "null argument");
  NX(cudaStreamSynchronize(h->stream));
  NX(cudaMemcpy(params, h->master, bxn::NP * 4, cudaMemcpyDeviceToHost));
  return BX_OK;
}

int bx_gnn_set_graph(bx_gnn_handle h, int n_nodes, const int32_t* ptr, const int32_t* nbr) {
  if (!h || !ptr || n_nodes <= 0) return nfail(BX_EINVAL, "bad graph arguments");
  const int nnz = ptr[n_nodes];
  if (ptr[0] != 0 || nnz < 0 || (nnz > 0 && !nbr)) return nfail(BX_EINVAL, "bad row pointers");
  std::vector<int> cnt(n_nodes + 1, 0);
  std::vector<float> inv(n_nodes, 0.f);
  for (int i = 0; i < n_nodes; ++i) {
    if (ptr[i + 1] < ptr[i]) return nfail(BX_EINVAL, "row pointers decrease");
    const int d = ptr[i + 1] - ptr[i];
    inv[i] = d > 0 ? 1.0f / (float)d : 0.f;
    for (int p = ptr[i]; p < ptr[i + 1]; ++p) {
      if (nbr[p] < 0 || nbr[p] >= n_nodes) return nfail(BX_EINVAL, "neighbour index out of range");
      cnt[nbr[p] + 1]++;
    }
  }
  for (int j = 0; j < n_nodes; ++j) cnt[j + 1] += cnt[j];
  std::vector<int> ptrT(cnt), nbrT(std::max(nnz, 1));
  std::vector<int> fill(cnt.begin(), cnt.end() - 1);
  for (int i = 0; i < n_nodes; ++i)
    for (int p = ptr[i]; p < ptr[i + 1]; ++p) nbrT[fill[nbr[p]]++] = i;
  void* old[] = {h->ptr, h->nbr, h->ptrT, h->nbrT, h->inv_deg};
  for (void* p : old) cudaFree(p);
  h->ptr = h->nbr = h->ptrT = h->nbrT = nullptr;
  h->inv_deg = nullptr;
  const size_t nz = (size_t)std::max(nnz, 1);
  if (cudaMalloc(&h->ptr, (size_t)(n_nodes + 1) * 4) != cudaSuccess || cudaMalloc(&h->nbr, nz * 4) != cudaSuccess ||
      cudaMalloc(&h->ptrT, (size_t)(n_nodes + 1) * 4) != cudaSuccess ||
      cudaMalloc(&h->nbrT, nz * 4) != cudaSuccess || cudaMalloc(&h->inv_deg, (size_t)n_nodes * 4) != cudaSuccess) {
    cudaGetLastError();
    return nfail(BX_ENOMEM, "cudaMalloc graph");
  }
  NX(cudaMemcpy(h->ptr, ptr, (size_t)(n_nodes + 1) * 4, cudaMemcpyHostToDevice));
  if (nnz > 0) NX(cudaMemcpy(h->nbr, nbr, (size_t)nnz * 4, cudaMemcpyHostToDevice));
  NX(cudaMemcpy(h->ptrT, ptrT.data(), (size_t)(n_nodes + 1) * 4, cudaMemcpyHostToDevice));
  NX(cudaMemcpy(h->nbrT, nbrT.data(), nz * 4, cudaMemcpyHostToDevice));
  NX(cudaMemcpy(h->inv_deg, inv.data(), (size_t)n_nodes * 4, cudaMemcpyHostToDevice));
  h->n_graph = n_nodes;
  h->h_ptr.assign(ptr, ptr + n_nodes + 1);
  h->h_nbr.assign(nbr, nbr + nnz);
  h->ok_lo = h->ok_hi = -1;
  return BX_OK;
}

int bx_gnn_forward(bx_gnn_handle h, int lo, int hi, const float* x, int n_in, float* y, int n_out) {
  if (!h || !x || !y || n_in <= 0 || n_in > W || n_out <= 0 || n_out > W)
    return nfail(BX_EINVAL, "bx_gnn_forward: bad arguments");
  int rc = check_range(h, lo, hi);
  if (rc != BX_OK) return rc;
  rc = forward(h, lo, hi, x, n_in, n_out);
  if (rc != BX_OK) return rc;
  NX(cudaMemcpyAsync(y, h->yhat, (size_t)(hi - lo) * n_out * 4, cudaMemcpyDeviceToDevice, h->stream));
  NX(cudaStreamSynchronize(h->stream));
  return check_tc(h);
}

int bx_gnn_gradients(bx_gnn_handle h, int lo, int hi, const float* x, int n_in, const float* y, int n_out,
                     float* grad_host, float* loss_host) {
  if (!h || !x || !y || !grad_host || n_in <= 0 || n_in > W || n_out <= 0 || n_out > W)
    return nfail(BX_EINVAL, "bx_gnn_gradients: bad arguments");
  int rc = check_range(h, lo, hi);
  if (rc == BX_OK) rc = forward(h, lo, hi, x, n_in, n_out);
  int nb = 0;
  if (rc == BX_OK) rc = backward(h, lo, hi, y, n_out, &nb);
  if (rc != BX_OK) return rc;
  bxn::k_update<false><<<kUpGrid, kUpThreads, 0, h->stream>>>(nb, h->part, n_out, h->loss_part,
                                                             1.0f / ((float)(hi - lo) * (float)n_out), h->loss, h->grad,
                                                             bxn::AdamArgs{});
  NX(cudaGetLastError());
  NX(cudaStreamSynchronize(h->stream));
  NX(cudaMemcpy(grad_host, h->grad, bxn::NP * 4, cudaMemcpyDeviceToHost));
  if (loss_host) NX(cudaMemcpy(loss_host, h->loss, 4, cudaMemcpyDeviceToHost));
  return check_tc(h);
}

int bx_gnn_train_step(bx_gnn_handle h, int lo, int hi, const float* x, int n_in, const float* y, int n_out, float lr,
                      float* loss_host) {
  if (!h || !x || !y || n_in <= 0 || n_in > W || n_out <= 0 || n_out > W || !(lr > 0.f))
    return nfail(BX_EINVAL, "bx_gnn_train_step: bad arguments");
  int rc = check_range(h, lo, hi);
  if (rc == BX_OK) rc = forward(h, lo, hi, x, n_in, n_out);
  int nb = 0;
  if (rc == BX_OK) rc = backward(h, lo, hi, y, n_out, &nb);
  if (rc != BX_OK) return rc;
  const float b1 = 0.9f, b2 = 0.999f;
  h->step += 1;
  const float bc1 = 1.f - powf(b1, (float)h->step), bc2 = 1.f - powf(b2, (float)h->step);
  bxn::k_update<true><<<kUpGrid, kUpThreads, 0, h->stream>>>(
      nb, h->part, n_out, h->loss_part, 1.0f / ((float)(hi - lo) * (float)n_out), h->loss, h->grad,
      bxn::AdamArgs{h->master, h->m, h->v, h->wb, lr, b1, b2, 1e-8f, bc1, bc2});
  NX(cudaGetLastError());
  if (loss_host) {
    unsigned r[2];                          // the loss and err
    NX(cudaMemcpyAsync(r, h->loss, 8, cudaMemcpyDeviceToHost, h->stream));
    NX(cudaStreamSynchronize(h->stream));
    std::memcpy(loss_host, &r[0], 4);
    if (r[1]) return nfail(BX_ECUDA, "network: a tensor-core wait timed out");
  }
  return BX_OK;
}

int bx_gnn_destroy(bx_gnn_handle h) {
  if (!h) return BX_OK;
  void* ptrs[] = {h->master, h->m, h->v, h->grad, h->wb, h->ptr, h->nbr, h->ptrT, h->nbrT, h->inv_deg,
                  h->act, h->yhat, h->dHa, h->dHb, h->Ga, h->Gb, h->part, h->loss_part, h->loss};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
  return BX_OK;
}

}  // extern "C"
