// bx_network.cuh -- the molecule / gene-regulatory-network step on the GPU.
//
// MasterOfNetworks.run_loop (chemistry/networks.py:2805-2983) for the
// substances of one network on a plain FP64 cluster without extracellular
// spaces, as two kernels per time step, one CTA per tile of up to 32 cells:
//
//   k_net_cell  per cell: Molecule.update_intra of every substance
//               (networks.py:5714-5807); growth/decay and cell-zone reaction
//               rates from the influencer tables (write_growth_and_decay,
//               write_reactions, get_influencers); c += (RM @ rates) dt; then
//               molecule_mover's membrane GHK flux and update_Co
//               (sim_toolbox.py:939-964, 1155-1207).  Writes the cell and
//               membrane values after the membrane step ("mid") and one
//               partial sum of flux * mem_sa per substance per CTA (the
//               auto-mixed environment, sim_toolbox.py:1196-1205).
//   k_net_gj    per cell: the gap-junction GHK flux (sim_toolbox.py:967-1000)
//               between the mid values of the membrane and its partner, the
//               final cell and membrane values and the negative-concentration
//               checks (sim_toolbox.py:1125-1151).  CTA 0 also reduces the
//               environment partials in a fixed order.
//
// Each kernel runs in phases over its tile, so that every phase has a lane for
// each independent value: a lane per (cell, substance or reaction) for the
// rates (a warp works on one table entry), a lane per membrane for the fluxes
// (coalesced loads), a lane per (cell, substance) for the sums over a cell's
// membranes, in membrane order.  A flux that is the same at all membranes of a
// cell is formed once.  Bound by the FP64 pipe and, before, by latency: with a
// thread per cell (4 warps an SM at 20k cells, strided membrane loads, the
// concentrations in local memory) 20,432 cells took 58 + 41 us, as written 31 + 20.
//
// The split into two launches is the one place the step needs every cell:
// the gap-junction flux reads the partner cell after its membrane step.
//
// Data layout in HBM (row = substance): c_cells [S][C], cc_at_mem [S][M] and
// their "mid" copies, the last step's fluxes f_mem/f_gj [S][M] and reaction
// rates [R][C], growth
// modulation [S][C] and target masks [S][C] only for the substances that have
// them, env [S], env partials [ntile][S]; the tables (substances, terms,
// reactions, stoichiometry) are one small block in global memory that every
// warp reads uniformly.  Geometry and Vmem are the cluster handle's own arrays.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "bx_env_np.cuh"
#include "bx_kernels.cuh"

namespace bx {

constexpr int kNetMaxSub = 16;
constexpr int kNetMaxReact = 32;
constexpr int kNetMaxTerms = 256;
constexpr int kNetStoich = 4;
constexpr int kNetTPB = 256;
constexpr int kNetCells = 32;           // most cells of a tile: a warp's lanes

enum NetTermKind { NT_ACT = 0, NT_ACT_INDEP = 1, NT_INH = 2, NT_DIRECT_POS = 3, NT_DIRECT_NEG = 4 };

struct NetTermD {
  int kind, sub, env, pad;
  double inv_km, n;        // 1 / Km (the host divides once)
};

struct NetSubD {
  double z, Dm, Do, Dgj, tdf, r_prod, r_decay, decay_max, inv_gsf;
  int growth, ui, gj_imp, gt0, gnt, dt0, dnt, mod_row, mask_row, pad;
};

struct NetReactD {
  int nr, np, r[kNetStoich], p[kNetStoich];
  double rc[kNetStoich], inv_rkm[kNetStoich], pc[kNetStoich];
  double vmax, inv_keq;    // inv_keq 0: no standard free energy
  int t0, nt;
};

// The tables, one block of plain data.
struct NetTables {
  int S, R, T, pad;
  NetSubD sub[kNetMaxSub];
  NetReactD react[kNetMaxReact];
  double rm[kNetMaxSub][kNetMaxReact];   // stoichiometry of the reactions (create_reaction_matrix)
  NetTermD term[kNetMaxTerms];
};

struct NetArgs {
  int C, M;
  double dt, inv_tm, F_RT, inv_gj_len, gj_block, inv_vol_env_M;
  // cluster geometry and state (the handle's arrays)
  const int* cell_ptr;
  const int* m2c;
  const int* nn;
  const int* nn_cell;
  const uint8_t* bflag;
  const double* mem_sa;
  const double* cell_vol;
  const double* gj_w;        // static weights (times gj_block: sim.gjopen)
  const double* gjo;         // gated open fraction, or nullptr
  const double* vm;          // Vmem the network reads (the start of the ion step)
  // network
  const NetTables* tab;
  const double* gamma;       // [M] mem_sa / ((3/4) mem_vol)
  const double* g_over_r;    // [M] gamma / R_rads
  const double* gmod;        // [rows][C]
  const uint8_t* gmask;      // [rows][C]
  double* c_cells;           // [S][C]
  double* cmem;              // [S][M]
  double* c_mid;             // [S][C]
  double* cmem_mid;          // [S][M]
  double* env;               // [S]
  double* env_part;          // [ntile][S]
  double* f_mem;             // [S][M] (OUT)
  double* f_gj;              // [S][M] (OUT)
  double* rates;             // [R][C] (OUT) cell-zone reaction rates (MasterOfNetworks.reaction_rates)
  unsigned long long* neg;   // negative concentrations seen
  int ntile, tile_cells;     // tiles of tile_cells cells (at most kNetCells)
  int tile_mems;             // most membranes of a tile
};

// sim_toolbox.electroflux (sim_toolbox.py:18-69) for a general charge, FP64,
// with Dk = Dc / d and zF = (z + 1e-25) F / (R T) hoisted out of the
// membrane loops, and the FP64 transcendentals only where they carry
// information (the GPU's FP64 pipe bounds these kernels):
//   |a| < 1e-17 (every neutral substance: a = 1e-25 v F/RT): exp(-a) rounds
//     to 1 and expm1(-a) to -a, in FP64 as in NumPy, so the flux is
//     -Dk (cB - cA) (a few ulp from BETSE's order of operations);
//   |a| > 1e-3: -expm1(-a) = 1 - exp(-a) to within 1e-13 relative;
//   otherwise (small gap-junction voltages) the Taylor series of expm1(-a)
//   to the fifth power, whose remainder a^6/720 is below 2e-21 |a|.
__device__ __forceinline__ bool net_neutral(double zF) { return fabs(zF) < 1.0e-20; }

// |x| against a power of ten through the exponent and upper mantissa bits (the
// FP64 compare costs a pipe slot): hi is the bound's upper word, and the
// formulas on both sides of each bound agree there.
__device__ __forceinline__ int net_abs_hi(double x) { return __double2hiint(x) & 0x7fffffff; }
constexpr int kHi1e17 = 0x3c670ef5;      // upper word of 1e-17
constexpr int kHi1e3 = 0x3f50624d;       // upper word of 1e-3
// x < 0, the compare itself only where the sign bit is set
__device__ __forceinline__ int net_is_neg(double x) { return __double2hiint(x) < 0 && x < 0.0 ? 1 : 0; }

// What a substance's fluxes need, formed once per CTA.
struct NetFlux {
  double zF, Dk, kq;                     // (z + 1e-25) F / (R T); D / d; membrane step: Do dt', junctions: dt'
  int on, neutral, ui, pad;              // on: the substance crosses
};

__device__ __forceinline__ double net_ghk(double cA, double cB, double Dk, double zF, bool neutral, double v) {
  if (neutral) return -Dk * (cB - cA);
  const double a = zF * (v + kNonce);
  const int aa = net_abs_hi(a);
  if (aa < kHi1e17) return -Dk * (cB - cA);
  double ea, den;
  if (aa > kHi1e3) {
    ea = exp(-a);
    den = 1.0 - ea;
  } else {
    const double x = -a;
    const double em1 = x * (1.0 + x * (0.5 + x * (1.0 / 6.0 + x * (1.0 / 24.0 + x * (1.0 / 120.0)))));
    ea = 1.0 + em1;
    den = -em1;
  }
  return -(Dk * a) * ((cB - cA * ea) / den);
}

// (c/Km)^n: BETSE's '**' (C pow); exponents 1 and 2 by multiplication (the
// same value as a correctly rounded pow), others by pow.
__device__ __forceinline__ double net_pow(double x, double n) {
  if (n == 1.0) return x;
  if (n == 2.0) return x * x;
  return pow(x, n);
}

// cs: the cell's concentrations, kNetCells apart
__device__ __forceinline__ double net_conc(const NetTermD& t, const double* cs, const double* env) {
  return t.env ? env[t.sub] : cs[t.sub * kNetCells];
}

// One influencer factor (get_influencers, networks.py:5084-5600).  The host
// orders a factor's terms as BETSE composes its string: multiplicative
// activators, independent activators, inhibitors, then the direct terms
// (activators' before inhibitors'), so one pass evaluates it in BETSE's
// operation order: ((a1*a2) + i1 + i2) * (h1*h2) * (d1 + d2 ...).
__device__ double net_factor(const NetTables& tb, int t0, int nt, const double* cs, const double* env) {
  double act = 1.0, inh = 1.0, dsum = 0.0;
  bool any_mult = false, any_inh = false, any_direct = false;
  for (int q = t0; q < t0 + nt; ++q) {
    const NetTermD& t = tb.term[q];
    const double c = net_conc(t, cs, env);
    switch (t.kind) {
      case NT_ACT: {
        const double x = net_pow(c * t.inv_km, t.n);
        const double h = x / (1.0 + x);
        act = any_mult ? act * h : h;
        any_mult = true;
        break;
      }
      case NT_ACT_INDEP: {
        const double x = net_pow(c * t.inv_km, t.n);
        act = act + x / (1.0 + x);
        break;
      }
      case NT_INH: {
        const double h = 1.0 / (1.0 + net_pow(c * t.inv_km, t.n));
        inh = any_inh ? inh * h : h;
        any_inh = true;
        break;
      }
      case NT_DIRECT_POS:
        dsum = any_direct ? dsum + c : c;
        any_direct = true;
        break;
      default:
        dsum = any_direct ? dsum - c : -c;
        any_direct = true;
        break;
    }
  }
  const double a = act * inh;
  return any_direct ? a * dsum : a;
}

// growth and decay of substance k (write_growth_and_decay)
__device__ __forceinline__ double net_growth(const NetArgs& a, const NetTables& tb, int k, int c, const double* cs,
                                             const double* env) {
  const NetSubD& sb = tb.sub[k];
  if (!sb.growth || !(sb.mask_row < 0 || a.gmask[(size_t)sb.mask_row * a.C + c])) return 0.0;
  const double mod = sb.mod_row < 0 ? 1.0 : a.gmod[(size_t)sb.mod_row * a.C + c];
  const double cc = cs[k * kNetCells] * sb.inv_gsf;
  const double ga = net_factor(tb, sb.gt0, sb.gnt, cs, env);
  const double da = net_factor(tb, sb.dt0, sb.dnt, cs, env);
  return mod * (sb.r_prod * sb.tdf) * ga - (sb.r_decay * sb.tdf) * cc - (sb.decay_max * sb.tdf) * da * cc;
}

// rate of reaction j (write_reactions)
__device__ __forceinline__ double net_rate(const NetTables& tb, int j, const double* cs, const double* env) {
  const NetReactD& rx = tb.react[j];
  const double al = net_factor(tb, rx.t0, rx.nt, cs, env);
  if (rx.inv_keq == 0.0) {
    double fwd = 1.0;
    for (int q = 0; q < rx.nr; ++q) {
      const double x = net_pow(cs[rx.r[q] * kNetCells] * rx.inv_rkm[q], rx.rc[q]);
      fwd = q == 0 ? x / (1.0 + x) : fwd * (x / (1.0 + x));
    }
    return rx.vmax * al * fwd;
  }
  // BETSE's quotient applies the power before the 1e-3 (networks.py:1364-1396)
  double num = 1.0, den = 1.0;
  for (int q = 0; q < rx.np; ++q) {
    const double t = 1.0e-3 * net_pow(cs[rx.p[q] * kNetCells], rx.pc[q]);
    num = q == 0 ? t : num * t;
  }
  for (int q = 0; q < rx.nr; ++q) {
    const double t = 1.0e-3 * net_pow(cs[rx.r[q] * kNetCells], rx.rc[q]);
    den = q == 0 ? t : den * t;
  }
  return rx.vmax * al * (1.0 - (num / den) * rx.inv_keq);
}

// dynamic shared memory of both kernels, in doubles
__host__ __device__ constexpr int net_smem_cell(int S, int R, int nm) { return (3 * S + R) * kNetCells + S * nm; }
__host__ __device__ constexpr int net_smem_gj(int S, int nm) { return S * kNetCells + S * nm; }

template <bool OUT>
__global__ void __launch_bounds__(kNetTPB) k_net_cell(NetArgs a) {
  // the tables are read in place: every lane of a warp reads the same entry,
  // one broadcast load from L1
  const NetTables& tb = *a.tab;
  extern __shared__ double ns[];
  __shared__ double env[kNetMaxSub], siv[kNetCells], sv[kNetCells];
  __shared__ NetFlux fx[kNetMaxSub];
  const int S = tb.S, R = tb.R, t = threadIdx.x, warp = t >> 5, lane = t & 31;
  double* cs = ns;                               // [S][32] concentrations
  double* sr = cs + S * kNetCells;               // [S + R][32] growth, reaction rates
  double* sf0 = sr + (S + R) * kNetCells;        // [S][32] membrane flux at the cell's Vmem
  double* sfa = sf0 + S * kNetCells;             // [S][tile_mems] flux times area
  const int c0 = blockIdx.x * a.tile_cells, nc = min(a.tile_cells, a.C - c0);
  const int m0 = a.cell_ptr[c0], nm = a.cell_ptr[c0 + nc] - m0;
  for (int q = t; q < S * kNetCells; q += kNetTPB) {
    const int k = q / kNetCells, lc = q - k * kNetCells;
    cs[q] = lc < nc ? a.c_cells[(size_t)k * a.C + c0 + lc] : 0.0;
  }
  if (t < S) {
    const NetSubD& sb = tb.sub[t];
    env[t] = a.env[t];
    const double zF = (sb.z + kNonce) * a.F_RT;
    fx[t] = NetFlux{zF, sb.Dm * a.inv_tm, sb.Do * (a.dt * sb.tdf), sb.Dm != 0.0, net_neutral(zF), sb.ui, 0};
  }
  if (warp == kNetTPB / 32 - 1 && lane < nc) {
    siv[lane] = 1.0 / a.cell_vol[c0 + lane];
    sv[lane] = a.vm[min(a.cell_ptr[c0 + lane], a.M - 1)];
  }
  __syncthreads();
  // rates on the concentrations at the start of the step; the membrane flux of
  // a substance whose membrane-side value is the cell's
  for (int j = warp; j < 2 * S + R; j += kNetTPB / 32) {
    if (lane >= nc) continue;
    const double* cl = cs + lane;
    if (j < S) {
      sr[j * kNetCells + lane] = net_growth(a, tb, j, c0 + lane, cl, env);
    } else if (j < S + R) {
      const double rate = net_rate(tb, j - S, cl, env);
      sr[j * kNetCells + lane] = rate;
      if (OUT) a.rates[(size_t)(j - S) * a.C + c0 + lane] = rate;
    } else {
      const int k = j - S - R;
      if (fx[k].on && !fx[k].ui)
        sf0[k * kNetCells + lane] = net_ghk(env[k], cl[k * kNetCells], fx[k].Dk, fx[k].zF, fx[k].neutral, sv[lane]);
    }
  }
  __syncthreads();
  int neg = 0;
  for (int ml = t; ml < nm; ml += kNetTPB) {
    const int m = m0 + ml, lc = a.m2c[m] - c0;
    const double sa = a.mem_sa[m], v = a.vm[m];
    const bool same = __double_as_longlong(v) == __double_as_longlong(sv[lc]);
    for (int k = 0; k < S; ++k) {
      const NetFlux& x = fx[k];
      const size_t km = (size_t)k * a.M + m;
      double f = 0.0;
      if (x.ui) {
        // Molecule.update_intra, implicit Euler toward the cell centre
        // (neutral substance: no field term); kq = gamma Do dt' / R_rads
        const double kq = a.g_over_r[m] * x.kq;
        double cm = (kq * cs[k * kNetCells + lc] + a.cmem[km]) / (1.0 + kq);
        neg += net_is_neg(cm);
        if (x.on) {
          f = net_ghk(env[k], cm, x.Dk, x.zF, x.neutral, v);
          sfa[k * a.tile_mems + ml] = f * sa;
          cm = cm + f * a.gamma[m] * a.dt;
        }
        a.cmem_mid[km] = cm;
      } else if (x.on) {
        f = same ? sf0[k * kNetCells + lc]
                 : net_ghk(env[k], cs[k * kNetCells + lc], x.Dk, x.zF, x.neutral, v);
        sfa[k * a.tile_mems + ml] = f * sa;
      }
      if (OUT) a.f_mem[km] = f;
    }
  }
  __syncthreads();
  for (int k = warp; k < S; k += kNetTPB / 32) {
    const bool on = fx[k].on;
    double s = 0.0;
    if (lane < nc) {
      const int c = c0 + lane;
      if (on)
        for (int ml = a.cell_ptr[c] - m0; ml < a.cell_ptr[c + 1] - m0; ++ml) s += sfa[k * a.tile_mems + ml];
      double delta = sr[k * kNetCells + lane];
      for (int j = 0; j < R; ++j) delta += tb.rm[k][j] * sr[(S + j) * kNetCells + lane];
      const double c1 = cs[k * kNetCells + lane] + delta * a.dt;
      a.c_mid[(size_t)k * a.C + c] = on ? c1 + (s * siv[lane]) * a.dt : c1;
    }
    if (on)
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) a.env_part[(size_t)blockIdx.x * S + k] = s;
  }
  if (neg) atomicAdd(a.neg, (unsigned long long)neg);
}

template <bool OUT>
__global__ void __launch_bounds__(kNetTPB) k_net_gj(NetArgs a) {
  const NetTables& tb = *a.tab;
  extern __shared__ double ns[];
  const int S = tb.S, t = threadIdx.x, warp = t >> 5, lane = t & 31;
  __shared__ double siv[kNetCells];
  __shared__ NetFlux fx[kNetMaxSub];
  double* sc = ns;                               // [S][32] concentrations, mid then final
  double* sfa = sc + S * kNetCells;              // [S][tile_mems] -flux times area
  const int c0 = blockIdx.x * a.tile_cells, nc = min(a.tile_cells, a.C - c0);
  const int m0 = a.cell_ptr[c0], nm = a.cell_ptr[c0 + nc] - m0;
  grid_wait();
  for (int q = t; q < S * kNetCells; q += kNetTPB) {
    const int k = q / kNetCells, lc = q - k * kNetCells;
    sc[q] = lc < nc ? a.c_mid[(size_t)k * a.C + c0 + lc] : 0.0;
  }
  if (t < S) {
    const NetSubD& sb = tb.sub[t];
    const double zF = (sb.z + kNonce) * a.F_RT;
    fx[t] = NetFlux{zF, sb.Dgj * a.gj_block * a.inv_gj_len, a.dt * sb.tdf, !sb.gj_imp, net_neutral(zF), sb.ui, 0};
  }
  if (warp == kNetTPB / 32 - 1 && lane < nc) siv[lane] = 1.0 / a.cell_vol[c0 + lane];
  __syncthreads();
  int neg = 0;
  for (int ml = t; ml < nm; ml += kNetTPB) {
    const int m = m0 + ml, lc = a.m2c[m] - c0, n = a.nn[m], cn = a.nn_cell[m];
    const bool open = !a.bflag[m];
    const double sa = a.mem_sa[m], dv = a.vm[n] - a.vm[m];
    const double go = a.gjo ? a.gjo[m] : a.gj_block * a.gj_w[m];
    for (int k = 0; k < S; ++k) {
      const NetFlux& x = fx[k];
      const size_t km = (size_t)k * a.M + m;
      double f = 0.0;
      if (x.on && open) {
        const double cA = x.ui ? a.cmem_mid[km] : sc[k * kNetCells + lc];
        const double cB = x.ui ? a.cmem_mid[(size_t)k * a.M + n] : a.c_mid[(size_t)k * a.C + cn];
        f = net_ghk(cA, cB, x.Dk * go, x.zF, x.neutral, dv);
      }
      if (x.on) sfa[k * a.tile_mems + ml] = -f * sa;
      if (x.ui) {
        double cm = a.cmem_mid[km];
        if (x.on) cm = cm + (-f) * a.gamma[m] * x.kq;
        a.cmem[km] = cm;
        neg += net_is_neg(cm);
      }
      if (OUT) a.f_gj[km] = f;
    }
  }
  __syncthreads();
  for (int k = warp; k < S; k += kNetTPB / 32) {
    if (lane >= nc) continue;
    const int c = c0 + lane;
    double c3 = sc[k * kNetCells + lane];
    if (fx[k].on) {
      double s = 0.0;
      for (int ml = a.cell_ptr[c] - m0; ml < a.cell_ptr[c + 1] - m0; ++ml) s += sfa[k * a.tile_mems + ml];
      c3 = c3 + (s * siv[lane]) * fx[k].kq;
      sc[k * kNetCells + lane] = c3;
    }
    a.c_cells[(size_t)k * a.C + c] = c3;
    neg += net_is_neg(c3);
  }
  __syncthreads();
  for (int ml = t; ml < nm; ml += kNetTPB) {
    const int m = m0 + ml, lc = a.m2c[m] - c0;
    for (int k = 0; k < S; ++k)
      if (!fx[k].ui) a.cmem[(size_t)k * a.M + m] = sc[k * kNetCells + lc];
  }
  if (blockIdx.x == 0) {
    // the auto-mixed environment: mean over membranes of env - f sa dt / vol_env
    for (int k = warp; k < S; k += kNetTPB / 32) {
      double s = 0.0;
      for (int b = lane; b < a.ntile; b += 32) s += a.env_part[(size_t)b * S + k];
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      if (lane == 0) {
        const double e = a.env[k] - (s * a.dt) * a.inv_vol_env_M;
        a.env[k] = e;
        if (e < 0.0) atomicAdd(a.neg, 1ull);
      }
    }
  }
  if (neg) atomicAdd(a.neg, (unsigned long long)neg);
}

}  // namespace bx
