// bx_env.cuh -- environment-grid kernels (extracellular spaces and fields).
//
// The grid is row-major (ny, nx), k = i*nx + j, as FiniteDiffSolver.cell_grid
// lays it out (betse/science/math/finitediff.py:158-250).  Each kernel is one
// thread per grid cell; the work is a few hundred bytes per cell, HBM- or
// launch-bound, and runs inside the step's CUDA graph.
#pragma once
#include "bx_env_np.cuh"
#include "bx_kernels.cuh"

namespace bx {

template <typename R>
__global__ void k_env_np_flux(EnvNp a) {
  env_np_flux<R>(a, blockIdx.x * blockDim.x + threadIdx.x);
}

// fd.diff with the reference's flipped one-sided edge signs (finitediff.py:1268-1303)
template <typename R = double>
__device__ __forceinline__ R ddx_neg(const R* f, const EnvConst& e, int i, int j) {
  // diff(-f, axis=0)
  const R* r = f + i * e.nx;
  const R inv_d = env_inv_d<R>(e), inv_2d = env_inv_2d<R>(e);
  if (j == 0) return ((-r[0]) - (-r[1])) * inv_d;
  if (j == e.nx - 1) return ((-r[j - 1]) - (-r[j])) * inv_d;
  return -((-r[j - 1]) - (-r[j + 1])) * inv_2d;
}
template <typename R = double>
__device__ __forceinline__ R ddy_neg(const R* f, const EnvConst& e, int i, int j) {
  // diff(-f, axis=1)
  const int nx = e.nx;
  const R inv_d = env_inv_d<R>(e), inv_2d = env_inv_2d<R>(e);
  if (i == 0) return -((-f[nx + j]) - (-f[j])) * inv_d;
  if (i == e.ny - 1) return -((-f[i * nx + j]) - (-f[(i - 1) * nx + j])) * inv_d;
  return -((-f[(i - 1) * nx + j]) - (-f[(i + 1) * nx + j])) * inv_2d;
}

// Environment charge of grid cell k from its new concentrations, for
// get_current's ECM branch (ion_current.py:82-92): rho = sum_i F z_i c_i (ions
// in order) and, on the membrane-touched cells, the surface-charge potential
// source v = (rho surf_scale) / (ko_env eo er); written by the kernel that
// produces the cell's final concentrations.
__device__ __forceinline__ void env_charge_out(int k, double rho, const uint8_t* touched, double* vsrc,
                                               double* rho_env, const EnvConst& e) {
  vsrc[k] = touched[k] ? (rho * e.surf_scale) * e.inv_koeoer : 0.0;
  if (rho_env) rho_env[k] = rho;
}

// tmp = cb + div(-f) dt (update_ecm sim.py:2247-2254), where the membrane
// exchange is a pass of its own.  One thread per (ion, grid cell).
__global__ void k_env_update(const double* __restrict__ cenv, double* tmp, const double* __restrict__ fx,
                             const double* __restrict__ fy, EnvConst e) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= e.I * e.G) return;
  const int ion = t / e.G, k = t - ion * e.G;
  const int i = k / e.nx, j = k - i * e.nx;
  const double* fxi = fx + (size_t)ion * e.G;
  const double* fyi = fy + (size_t)ion * e.G;
  const double div = ddx_neg(fxi, e, i, j) + ddy_neg(fyi, e, i, j);
  tmp[(size_t)ion * e.G + k] = cb_at(cenv, e, ion, i, j) + div * e.dt;
}

// The environment charge of each grid cell from its final concentrations
// (ions in order), for get_current's ECM branch.
__global__ void k_env_charge(const double* __restrict__ cenv, const uint8_t* __restrict__ touched, double* vsrc,
                             double* rho_env, EnvConst e) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= e.G) return;
  double rho = 0.0;
  for (int ion = 0; ion < e.I; ++ion) rho += e.zF[ion] * cenv[(size_t)ion * e.G + k];
  env_charge_out(k, rho, touched, vsrc, rho_env, e);
}

// fd.integrator (finitediff.py:1479-1512) of grid value k of one ion
__device__ __forceinline__ double env_integrate(const double* P, const EnvConst& e, int k) {
  const int i = k / e.nx, j = k - i * e.nx;
  if (on_edge(i, j, e.ny, e.nx)) return P[k];
  const double sides = (1 - e.sharpness) / 4;
  double F = e.sharpness * P[k];
  F += sides * P[k + e.nx];
  F += sides * P[k - e.nx];
  F += sides * P[k + 1];
  F += sides * P[k - 1];
  return F;
}

// The membrane exchange of one ion over rows [q0, q1), four at a time (their
// loads are independent), added in list order; a cell's lanes read a row together
__device__ __forceinline__ double env_exchange(const double* __restrict__ mem_flux_sa, int q0, int q1, int ion) {
  double s = 0.0;
  for (; q0 < q1; q0 += 4) {
    double fv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) fv[u] = q0 + u < q1 ? mem_flux_sa[(size_t)(q0 + u) * kMfs + ion] : 0.0;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (q0 + u < q1) s += -fv[u];
  }
  return s;
}

// The smoothed grid, where the membrane exchange is a later pass.  One thread
// per (ion, grid cell).
__global__ void k_env_integrate(double* out, const double* __restrict__ tmp, EnvConst e) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= e.I * e.G) return;
  const int ion = t / e.G, k = t - ion * e.G;
  out[t] = env_integrate(tmp + (size_t)ion * e.G, e, k);
}

// The membrane exchange onto an environment already advanced by the
// Nernst-Planck update: update_Co's ECM term (sim_toolbox.py:1185-1200), the
// same arithmetic as the fused kernels.  INTEGRATE: src is smoothed on the way
// (sharpness < 1).  kEnvUpCells grid cells per CTA, a lane per (cell, ion) with
// the ions contiguous, which read an exchange row together (by itself, 20,000
// cells on 200 x 200: 10.0 us; a thread per ion and cell in grid order, row after
// row, 11.8).
constexpr int kEnvUpT = 192, kEnvUpCells = 32;
template <bool INTEGRATE>
__global__ void __launch_bounds__(kEnvUpT) k_env_scatter(double* cenv, const double* __restrict__ src,
                                                         const int* __restrict__ env_ptr,
                                                         const double* __restrict__ mem_flux_sa, EnvConst e) {
  const int k0 = blockIdx.x * kEnvUpCells, nk = min(kEnvUpCells, e.G - k0);
  for (int q = threadIdx.x; q < nk * e.I; q += kEnvUpT) {
    const int lk = q / e.I, ion = q - lk * e.I, k = k0 + lk;
    const double s = env_exchange(mem_flux_sa, env_ptr[k], env_ptr[k + 1], ion);
    const double* P = src + (size_t)ion * e.G;
    const double F = INTEGRATE ? env_integrate(P, e, k) : P[k];
    cenv[(size_t)ion * e.G + k] = F + (s * e.inv_h_d2) * e.dt;
  }
}

// get_current ECM branch (ion_current.py:79-110): the axis-0 pass of a
// sigma=1 Gaussian with zero padding (scipy mode='constant') over the
// potential source the concentration kernel left in vsrc.
__global__ void k_env_gauss_y(const double* __restrict__ vsrc, double* tmp, EnvConst e) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= e.G) return;
  const int i = k / e.nx, j = k - i * e.nx;
  double acc = 0.0;
#pragma unroll
  for (int q = -4; q <= 4; ++q) {
    const int ii = i + q;
    if (ii < 0 || ii >= e.ny) continue;
    acc += e.gw[q + 4] * vsrc[ii * e.nx + j];
  }
  tmp[k] = acc;
}

// axis-1 pass of the Gaussian (+ Phi_b) -> v_env
__global__ void k_env_gauss_x(const double* __restrict__ tmp, const double* __restrict__ phib,
                              double* venv, EnvConst e) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= e.G) return;
  const int i = k / e.nx, j = k - i * e.nx;
  double acc = 0.0;
  for (int q = -4; q <= 4; ++q) {
    const int jj = j + q;
    if (jj < 0 || jj >= e.nx) continue;
    acc += e.gw[q + 4] * tmp[i * e.nx + jj];
  }
  venv[k] = acc + (phib ? phib[k] : 0.0);
}

// E = -gradient(scale * F)  (fd.gradient, finitediff.py:1236-1266)
// (and its FP32 copy in the split form)
__global__ void k_env_neg_grad(const double* __restrict__ F, double scale, double* Ex, double* Ey, float* Ex_f,
                               float* Ey_f, EnvConst e) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= e.G) return;
  const int i = k / e.nx, j = k - i * e.nx;
  const int nx = e.nx;
  auto f = [&](int a, int bb) { return scale * F[a * nx + bb]; };
  double gx, gy;
  if (j == 0) gx = (f(i, 1) - f(i, 0)) * e.inv_delta;
  else if (j == nx - 1) gx = (f(i, j) - f(i, j - 1)) * e.inv_delta;
  else gx = -(f(i, j - 1) - f(i, j + 1)) * e.inv_2delta;
  if (i == 0) gy = (f(1, j) - f(0, j)) * e.inv_delta;
  else if (i == e.ny - 1) gy = (f(i, j) - f(i - 1, j)) * e.inv_delta;
  else gy = -(f(i - 1, j) - f(i + 1, j)) * e.inv_2delta;
  Ex[k] = -gx;
  Ey[k] = -gy;
  if (Ex_f) {
    Ex_f[k] = (float)-gx;
    Ey_f[k] = (float)-gy;
  }
}

// ---------------------------------------------------------------------------
// Fused forms of the sequences above, for the common configuration (no
// Ca-ATPase, sharpness >= 1): fewer launches on a grid that is small against
// the GPU, the same arithmetic term by term.
// ---------------------------------------------------------------------------

// The concentration update, the membrane exchange and the environment charge
// in one launch: kEnvUpCells grid cells per CTA, a lane per (cell, ion) with the
// ions of a cell contiguous.  Each lane advances its ion's concentration in
// place (it reads only fluxes and its own cell's value); then a lane per cell
// adds F z_i c_i over the ions in order.
// R = float (split form): the divergence of the FP32 fluxes in FP32; the
// concentration, the membrane exchange and the charge stay FP64.
// Bound by the FP64 pipe in both forms, so what counts is full lanes: with
// eight lanes a cell and the charge summed by shuffles in all of them, 20 FP64
// warp instructions per four cells took 24 us (split) and 22 us (FP64) on
// 200 x 200 cells; as written 11.5 and 13 us (a launch by itself; split with the
// fluxes and constants converted from FP64 by every thread 15.0).
template <typename R>
__global__ void __launch_bounds__(kEnvUpT) k_env_update_charge(double* cenv, const R* __restrict__ fx,
                                                               const R* __restrict__ fy,
                                                               const int* __restrict__ env_ptr,
                                                               const double* __restrict__ mem_flux_sa,
                                                               const uint8_t* __restrict__ touched, double* vsrc,
                                                               double* rho_env, EnvConst e) {
  __shared__ double zc[kEnvUpCells * kMaxIons];
  grid_wait();
  const int k0 = blockIdx.x * kEnvUpCells, nk = min(kEnvUpCells, e.G - k0);
  for (int q = threadIdx.x; q < nk * e.I; q += kEnvUpT) {
    const int lk = q / e.I, ion = q - lk * e.I, k = k0 + lk;
    const int i = k / e.nx, j = k - i * e.nx;
    const R* fxi = fx + (size_t)ion * e.G;
    const R* fyi = fy + (size_t)ion * e.G;
    const R div = ddx_neg<R>(fxi, e, i, j) + ddy_neg<R>(fyi, e, i, j);
    double c = cb_at(cenv, e, ion, i, j) + (double)(div * env_dt<R>(e));
    const double s = env_exchange(mem_flux_sa, env_ptr[k], env_ptr[k + 1], ion);
    c = c + (s * e.inv_h_d2) * e.dt;
    cenv[(size_t)ion * e.G + k] = c;
    zc[q] = e.zF[ion] * c;
  }
  __syncthreads();
  if (threadIdx.x < nk) {
    double rho = 0.0;
    for (int q = 0; q < e.I; ++q) rho += zc[threadIdx.x * e.I + q];
    env_charge_out(k0 + threadIdx.x, rho, touched, vsrc, rho_env, e);
  }
  grid_release();
}

// k_env_gauss_y, k_env_gauss_x (+ Phi_b) and k_env_neg_grad in one launch:
// each CTA computes a kEnvTX x kEnvTY tile of E_env (and v_env) from the
// potential source in shared memory, with the halos the two Gaussian passes
// (4 cells) and the gradient (1 cell) need.
constexpr int kEnvTX = 32, kEnvTY = 16;
constexpr int kEnvVX = kEnvTX + 2, kEnvVY = kEnvTY + 2;        // v_env tile (gradient halo)
constexpr int kEnvSX = kEnvVX + 8, kEnvSY = kEnvVY + 8;        // source tile (Gaussian halo)
// R = float (split form): both passes and the gradient in FP32.
template <typename R>
__global__ void __launch_bounds__(kEnvTX * kEnvTY) k_env_fields_tile(const double* __restrict__ vsrc,
                                                                     const double* __restrict__ phib,
                                                                     double* venv, double scale, double* Ex,
                                                                     double* Ey, float* Ex_f, float* Ey_f, EnvConst e,
                                                                     int ntx) {
  __shared__ R src[kEnvSY][kEnvSX];
  __shared__ R gy[kEnvVY][kEnvSX];
  __shared__ R v[kEnvVY][kEnvVX];
  grid_wait();
  const int by = blockIdx.x / ntx, bx_ = blockIdx.x - by * ntx;
  const int i0 = by * kEnvTY - 1 - 4, j0 = bx_ * kEnvTX - 1 - 4;   // src tile origin
  const int nt = blockDim.x;
  for (int q = threadIdx.x; q < kEnvSY * kEnvSX; q += nt) {
    const int a = q / kEnvSX, b = q - a * kEnvSX, i = i0 + a, j = j0 + b;
    src[a][b] = (i >= 0 && i < e.ny && j >= 0 && j < e.nx) ? (R)vsrc[i * e.nx + j] : (R)0;
  }
  __syncthreads();
  // axis-0 pass (zero padding: taps outside the grid are skipped, as k_env_gauss_y does)
  for (int q = threadIdx.x; q < kEnvVY * kEnvSX; q += nt) {
    const int a = q / kEnvSX, b = q - a * kEnvSX, i = i0 + 4 + a;
    R acc = 0;
#pragma unroll
    for (int w = -4; w <= 4; ++w) {
      const int ii = i + w;
      if (ii < 0 || ii >= e.ny) continue;
      acc += env_gw<R>(e, w + 4) * src[a + 4 + w][b];
    }
    gy[a][b] = acc;
  }
  __syncthreads();
  // axis-1 pass + Phi_b -> v_env on the tile and its one-cell halo
  for (int q = threadIdx.x; q < kEnvVY * kEnvVX; q += nt) {
    const int a = q / kEnvVX, b = q - a * kEnvVX, i = i0 + 4 + a, j = j0 + 4 + b;
    R acc = 0;
    for (int w = -4; w <= 4; ++w) {
      const int jj = j + w;
      if (jj < 0 || jj >= e.nx) continue;
      acc += env_gw<R>(e, w + 4) * gy[a][b + 4 + w];
    }
    const bool in = i >= 0 && i < e.ny && j >= 0 && j < e.nx;
    v[a][b] = in ? acc + (phib ? (R)phib[i * e.nx + j] : (R)0) : (R)0;
  }
  __syncthreads();
  // E = -gradient(scale * v_env), one-sided on the grid edges
  const int a = threadIdx.x / kEnvTX + 1, b = threadIdx.x % kEnvTX + 1;
  const int i = by * kEnvTY + a - 1, j = bx_ * kEnvTX + b - 1;
  if (i >= e.ny || j >= e.nx) return;   // (an exited thread has released)
  const int k = i * e.nx + j;
  venv[k] = (double)v[a][b];
  const R sc = (R)scale, inv_d = env_inv_d<R>(e), inv_2d = env_inv_2d<R>(e);
  auto f = [&](int da, int db) { return sc * v[a + da][b + db]; };
  R gx, gyy;
  if (j == 0) gx = (f(0, 1) - f(0, 0)) * inv_d;
  else if (j == e.nx - 1) gx = (f(0, 0) - f(0, -1)) * inv_d;
  else gx = -(f(0, -1) - f(0, 1)) * inv_2d;
  if (i == 0) gyy = (f(1, 0) - f(0, 0)) * inv_d;
  else if (i == e.ny - 1) gyy = (f(0, 0) - f(-1, 0)) * inv_d;
  else gyy = -(f(-1, 0) - f(1, 0)) * inv_2d;
  Ex[k] = (double)(-gx);
  Ey[k] = (double)(-gyy);
  if (sizeof(R) == 4) {
    Ex_f[k] = (float)-gx;
    Ey_f[k] = (float)-gyy;
  }
  grid_release();
}

// ---------------------------------------------------------------------------
// Dense FP64 products Y[n x R] = A[n x n] X[n x R], R <= 4 (row-major).
// One warp per row; the row streams from HBM with 16-byte loads, X is
// L2-resident.  The HBM-bound form of np.dot(lapENVinv, .).
// ---------------------------------------------------------------------------
template <int R>
__global__ void __launch_bounds__(256) k_dense_rows(const double* __restrict__ A, const double* __restrict__ X,
                                                    double* __restrict__ Y, int n) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= n) return;
  const double* row = A + (size_t)warp * n;
  double acc[R];
#pragma unroll
  for (int r = 0; r < R; ++r) acc[r] = 0.0;
  const bool al16 = ((reinterpret_cast<uintptr_t>(row) & 15) == 0);
  int k0 = 0;
  if (al16) {
    const int n2 = n >> 1;
    const double2* row2 = reinterpret_cast<const double2*>(row);
    for (int q = lane; q < n2; q += 32) {
      const double2 a = __ldcs(row2 + q);
      const int kk = 2 * q;
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r] += a.x * X[(size_t)kk * R + r] + a.y * X[(size_t)(kk + 1) * R + r];
    }
    k0 = 2 * n2;
  }
  for (int kk = k0 + lane; kk < n; kk += 32) {
    const double a = row[kk];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] += a * X[(size_t)kk * R + r];
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const double s = warp_sum(acc[r]);
    if (lane == 0) Y[(size_t)warp * R + r] = s;
  }
}

}  // namespace bx
