// bx_env_np.cuh -- the extracellular grid's constants and Nernst-Planck flux,
// shared by the grid kernels and the step kernels that compute it beside
// their tiles.
#pragma once
#include "bx_kernels.cuh"

namespace bx {

// Programmatic dependent launch: grid_wait orders this kernel after the one
// before it; grid_release lets the next one start.  The kernels of a step with
// extracellular spaces release at their end: released at the start, the next
// kernel's CTAs fill whatever SMs have room and the FP64-bound ones end up with
// too many (20,400 cells on 200 x 200, FP64: 69 us a step instead of 59).
__device__ __forceinline__ void grid_wait() {
#if defined(__CUDA_ARCH__) && (__CUDA_ARCH__ >= 900)
  cudaGridDependencySynchronize();
#endif
}
__device__ __forceinline__ void grid_release() {
#if defined(__CUDA_ARCH__) && (__CUDA_ARCH__ >= 900)
  cudaTriggerProgrammaticLaunchCompletion();
#endif
}

struct EnvConst {
  int I, ny, nx, G;
  double delta, inv_delta, inv_2delta, dt, sharpness;
  double np_alpha[kMaxIons];   // z q / (kb T)  (times D_env per cell)
  double zF[kMaxIons];
  double c_bound[kMaxIons];
  double surf_scale;           // cell_height delta^2 / mean(memSa_per_envSquare[map])
  double inv_koeoer;           // 1 / (ko_env eo er)
  double screen;               // (2/(ko_env delta)) (cell_radius/true_cell_size)
  double inv_h_d2;             // 1 / (cell_height delta^2)
  double gw[9];                // Gaussian taps, sigma 1, radius 4
  // the split form's, rounded once: a conversion takes a slot of the FP64 pipe
  float inv_delta_f, inv_2delta_f, dt_f, np_alpha_f[kMaxIons], gw_f[9];
};
template <typename R> __device__ __forceinline__ R env_inv_d(const EnvConst& e) { return sizeof(R) == 4 ? (R)e.inv_delta_f : (R)e.inv_delta; }
template <typename R> __device__ __forceinline__ R env_inv_2d(const EnvConst& e) { return sizeof(R) == 4 ? (R)e.inv_2delta_f : (R)e.inv_2delta; }
template <typename R> __device__ __forceinline__ R env_dt(const EnvConst& e) { return sizeof(R) == 4 ? (R)e.dt_f : (R)e.dt; }
template <typename R> __device__ __forceinline__ R env_np_alpha(const EnvConst& e, int i) { return sizeof(R) == 4 ? (R)e.np_alpha_f[i] : (R)e.np_alpha[i]; }
template <typename R> __device__ __forceinline__ R env_gw(const EnvConst& e, int q) { return sizeof(R) == 4 ? (R)e.gw_f[q] : (R)e.gw[q]; }

__device__ __forceinline__ bool on_edge(int i, int j, int ny, int nx) {
  return i == 0 || j == 0 || i == ny - 1 || j == nx - 1;
}

// Boundary-set concentration (update_ecm sets the four edges, sim.py:2214-2217)
__device__ __forceinline__ double cb_at(const double* c, const EnvConst& e, int ion, int i, int j) {
  return on_edge(i, j, e.ny, e.nx) ? e.c_bound[ion] : c[(size_t)ion * e.G + i * e.nx + j];
}

// Nernst-Planck flux on the grid (update_ecm, sim.py:2219-2242;
// stb.nernst_planck_flux, sim_toolbox.py:385-413) with fd.gradient
// (finitediff.py:1236-1266).  E_env is the previous update_V's field.
// The grid kernels multiply by 1/delta and 1/(2 delta) where the reference
// divides (a difference of at most one rounding): an FP64 division costs
// GB300 several FP64-pipe operations, and the stencils are otherwise cheap.
// R = float is the split form's stencil: the concentration differences are
// taken in FP64 (the state) and scaled, with the drift term, in FP32.
// One thread per (ion, grid cell): t = ion*G + k.
struct EnvNp {
  const double *cenv, *Denv, *Ex, *Ey;
  double *fx, *fy;         // (split form in a step kernel's launch: written when a caller will read them)
  // split form: the same values in FP32, what the stencils use (null in FP64).
  // Converting them from FP64 in every thread cost the pipe more than the
  // stencils: a split step of 20,432 cells on 200 x 200 30.7 -> 22.9 us.
  const float *Denv_f, *Ex_f, *Ey_f;
  float *fx_f, *fy_f;
  EnvConst e;
  int nblk;                // blocks of a step kernel's launch that do this (0: a launch of its own)
};
template <typename R>
__device__ __forceinline__ void env_np_flux(const EnvNp& a, int t) {
  const EnvConst& e = a.e;
  if (t >= e.I * e.G) return;
  const int ion = t / e.G, k = t - ion * e.G;
  const int i = k / e.nx, j = k - i * e.nx;
  const double c0 = cb_at(a.cenv, e, ion, i, j);
  const R inv_d = env_inv_d<R>(e), inv_2d = env_inv_2d<R>(e);
  R gcx, gcy;
  if (j == 0) gcx = (R)(cb_at(a.cenv, e, ion, i, 1) - c0) * inv_d;
  else if (j == e.nx - 1) gcx = (R)(c0 - cb_at(a.cenv, e, ion, i, j - 1)) * inv_d;
  else gcx = -(R)(cb_at(a.cenv, e, ion, i, j - 1) - cb_at(a.cenv, e, ion, i, j + 1)) * inv_2d;
  if (i == 0) gcy = (R)(cb_at(a.cenv, e, ion, 1, j) - c0) * inv_d;
  else if (i == e.ny - 1) gcy = (R)(c0 - cb_at(a.cenv, e, ion, i - 1, j)) * inv_d;
  else gcy = -(R)(cb_at(a.cenv, e, ion, i - 1, j) - cb_at(a.cenv, e, ion, i + 1, j)) * inv_2d;
  const size_t o = (size_t)ion * e.G + k;
  constexpr bool F = sizeof(R) == 4;
  const R D = F ? (R)a.Denv_f[o] : (R)a.Denv[o];
  const R alpha = D * env_np_alpha<R>(e, ion);
  const R gvx = F ? -(R)a.Ex_f[k] : -(R)a.Ex[k], gvy = F ? -(R)a.Ey_f[k] : -(R)a.Ey[k];
  const R fx = -D * gcx - alpha * gvx * (R)c0, fy = -D * gcy - alpha * gvy * (R)c0;
  if (F) {
    a.fx_f[o] = (float)fx;
    a.fy_f[o] = (float)fy;
  }
  if (!F || a.fx) {
    a.fx[o] = (double)fx;
    a.fy[o] = (double)fy;
  }
}
// Membrane exchange f*sa: rows of kMfs values (ion contiguous), the membranes
// of a grid cell in consecutive rows (row env_ptr[k] + its rank), so that a
// grid cell reads one run of memory.
constexpr int kMfs = 8;

}  // namespace bx
