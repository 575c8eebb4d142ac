// bx_plain.cuh -- the plain FP64 step, factored per cell and per junction.
//
// GB300's FP64 pipe (one warp instruction in ~19 cycles per SM) bounds the
// plain form, so the kernel is built around how few FP64 instructions a step
// needs.  Without extracellular spaces, Phi_b and polarizability every
// membrane of a cell sees the same Vmem, the same membrane-side
// concentrations and the same environment.  So, exactly as real numbers:
//   * the transmembrane GHK flux of membrane m is Dm_i(m) times one factor
//     H_i per cell, and the Na/K and Ca pumps are one rate per cell:
//       sum_m f_i(m) sa(m) = H_i sum_m Dm_i(m) sa(m) + f_pump,i sum_m sa(m);
//   * the gap-junction flux through membrane m is w(m) D_i Q_i with Q_i
//     antisymmetric under swapping the two cells (expm1(a) = -expm1(-a) /
//     exp(-a)), so the two membranes of a junction share one evaluation.
// A cell with six membranes needs one set of exponentials and the pump once,
// and three junctions, where k_cell_step (bx_kernels.cuh) needs six of each:
// about 400 FP64 thread instructions a cell against 1900.  Everything stays
// FP64; only the order of the sums differs (one rounding per term).
// Measured per step (k_cell_step with k_env_mix before): 100k cells 403 ->
// 91 us, 20k cells 85 -> 30.4 us, 2900 cells 41 -> 10.1 us, 185 cells
// 40 -> 9.7 us (12.5 with the one-lane-per-ion kernel that this one replaced).
//
// One CTA advances one tile: NC consecutive cells of one cluster, in phases
// separated by bar.sync:
//   A  lane per junction ("entry"): the shared exponentials and Q of every ion;
//      lane per cell: the shared exponentials and the pumps
//   G  (voltage-gated junctions) lane per membrane: the open fraction, once
//      per ion as BETSE updates it
//   C  lane per (cell, ion): the segment sum over the cell's junctions, the
//      transmembrane sum and the concentration update
//   D  lane per cell: charge and Vmem; warp per ion: the tile's part of the
//      environment exchange
// Entries whose partner cell lies in the tile serve both sides; a halo entry
// (partner in another tile) is evaluated by both tiles.
//
// The environment sum runs over a binary tree of the cluster's cell indices
// (aligned powers of two, missing leaves zero), so its rounding depends
// neither on the tile size nor on what else is in a batch (NC is a power of two).
//
// Two launches of the same body (build_plain_layout chooses):
//   streaming   one step per launch (programmatic dependent launch); the last
//               tile of every 32 adds their parts, the last such group of the
//               cluster the groups' (ticket counters), and mixes the environment
//   (extracellular spaces: streaming, one launch a step before the grid's own,
//   without the environment sum.  The environment differs from membrane to
//   membrane, so a phase M, lane per membrane, gathers it and evaluates the
//   pump, and phase C forms each membrane's flux from two factors per cell and
//   ion, f sa = Dm sa (P - Q c_env): five FP64 instructions a membrane and ion.
//   The last blocks of the launch compute the grid's Nernst-Planck flux.
//   20,400 cells on 200 x 200: step 126 -> 57 us; 4975 on 100 x 100: 44 -> 27)
//   resident    many steps per cooperative launch, one tile per CTA, all of
//               them co-resident: the state stays in shared memory, tiles
//               exchange Vmem and concentrations through L2 and meet once a
//               step at a bounded grid barrier; the cells' own exponentials
//               and the junctions inside the tile are evaluated while the
//               barrier completes.
#pragma once
#include "bx_env_np.cuh"
#include "bx_kernels.cuh"
#include "bx_sync.cuh"

namespace bx {

constexpr int kPlainT = 256;            // threads per CTA
constexpr int kPlainNone = INT32_MIN;   // mem_ent: no junction
constexpr int kPlainRows = 8;           // resident: most rows of 32 tiles (the environment tree adds eight)

struct PlainGeom {
  int C, M, ntile;
  const int2* tile;        // [ntile] {first cell, cells}
  const int* tile_cl;      // [ntile] cluster
  const int* cl_tile;      // [ncl + 1] first tile of each cluster
  const int* cl_group;     // [ncl + 1] first group (of 32 tiles) of each cluster
  const int* ent_ptr;      // [ntile + 1] entries of each tile
  const int* n_local;      // [ntile] of them, those whose partner is in the tile (they come first)
  const int4* ent;         // {own cell (in the tile), partner cell (in the tile; halo: global), partner's first membrane, 0}
  const int* mem_ent;      // [M] the membrane's entry in its tile, ~entry on the partner's side, kPlainNone on the boundary
  const int* mem_gate;     // [M] (gated) entry whose |vgj| gates the membrane
  const int* cell_ptr;     // [C + 1]
  const int* m2c;          // [M]
  const double* mem_w;     // [M] gj_weight * mem_sa
  const double* mem_sa;    // [M]
  const double* dsa;       // [I][C] sum of Dm_i * mem_sa over the cell's membranes (ECM: [M][I] Dm_i * mem_sa)
  const double* sa;        // [C] sum of mem_sa
  const double* ivol;      // [C] 1 / cell_vol
  const double* diviterm;  // [C]
  const int* map_env;      // [M] (ECM)
  const int* env_slot;     // [M] (ECM) row of the exported f*sa
  int G;
};

struct PlainRun {
  double* vm[2];           // Vmem [M], read from [0] first
  double* ccm[2];          // membrane-side concentrations [I][C]
  int n_steps;             // resident: steps of this launch
  int nc_max, ne_max, nm_max;   // largest tile: cells, entries, membranes (shared memory)
  double* part;            // [ntile][I] tile parts of the environment exchange (resident: two copies)
  double* gpart;           // [groups + ...][I] group parts and the levels above them
  unsigned* ticket;        // [groups + ncl] zero between steps
  double* cenv;            // [ncl][I]
  const double* env_scale; // [ncl]
  unsigned* ctl;           // resident: barrier counter, timeout flag
  long long timeout_ns;
};

// Shared memory of one CTA, in doubles, for the largest tile.
constexpr int kPlainCell = 9;           // doubles of a cell's shared factors
struct PlainSmem {
  int q, v, cm, cc, x, s1, k, env, lvl, ga, gg, en, pm, total;
  __host__ __device__ PlainSmem(int nc, int ne, int nm, int I, bool gated, bool ecm) {
    int o = 0;
    auto take = [&](int n) { const int at = o; o += n; return at; };
    q = take(ne * I);
    v = take(nc);
    cm = take(nc * I);
    cc = take(nc * I);
    x = take(nc * I);
    s1 = take(nc * I);
    k = take(nc * kPlainCell);
    env = take(kMaxIons);
    lvl = take(8 * kPlainRows);
    ga = take(gated ? 2 * ne : 0);
    gg = take(gated ? nm * I : 0);
    en = take(ecm ? nm * I : 0);
    pm = take(ecm ? nm : 0);
    total = o;
  }
};
enum PlainCell { PK_K1 = 0, PK_E1, PK_K2, PK_E2, PK_FNA, PK_DTV, PK_FCA, PK_PC, PK_PR };   // kPlainCell rows

// BETSE's six-ion set as constants (ZP = 1) or the parameters' ions (ZP = 0)
template <int ZP> struct PlainIons {
  __device__ static int n(const StepConst& k) { return k.I; }
  __device__ static int zc(const StepConst& k, int i) { return k.zcode[i]; }
  static constexpr int NI = kMaxIons;
};
template <> struct PlainIons<1> {
  __device__ static constexpr int n(const StepConst&) { return 6; }
  __device__ static constexpr int zc(const StepConst&, int i) { return i < 2 ? 1 : i == 3 ? 2 : -1; }
  static constexpr int NI = 6;
};

// expm1 and exp by table (P. T. P. Tang, "Table-driven implementation of the
// exponential function in IEEE floating-point arithmetic", ACM TOMS 15, 1989;
// "... of the expm1 function ...", ACM TOMS 18, 1992): x = (64 m + j) ln2 / 64
// + r, |r| <= ln2 / 128, exp(x) = 2^m 2^(j/64) (1 + p), p = expm1(r) by its
// Taylor series to r^6 (the next term is below 2^-57 of p).  A table entry is
// 2^(j/64) rounded and the rest relative to it, so that
// expm1(x) = T (p + rest) + (T - 1).  Fourteen FP64 instructions, where the pipe
// spends 21.5 on expm1 and 16.8 on exp; outside |x| < 690 (and for NaN) those
// are called.  Against 113-bit values over 2 M points of |x| < 690, 10, 0.7,
// 0.02 and down to 1e-30: at most 1.12 ulp (expm1 1.14; below 0.02 alone 1.12
// and 0.51) and 0.51 ulp (exp 0.87).  A step of 100,043 cells 100.1 -> 91.4 us,
// of 185 cells 10.3 -> 9.7, voltage-gated 2,878 cells 18.2 -> 16.3.
constexpr double kLn2Hi = 0x1.62e42fefa0000p-7, kLn2Lo = 0x1.cf79abc9e3b3ap-46;   // ln2 / 64: 36 bits (times 17-bit integers exact) and the rest
constexpr double kInvLn2 = 0x1.71547652b82fep+6;                            // 64 / ln2
__device__ const double2 kExpTab[64] = {
    {0x1.0000000000000p+0, 0x0.0p+0}, {0x1.02c9a3e778061p+0, -0x1.160139cd8dc5dp-56},
    {0x1.059b0d3158574p+0, 0x1.cd2523567f613p-55}, {0x1.0874518759bc8p+0, 0x1.0f74e61e6c861p-57},
    {0x1.0b5586cf9890fp+0, 0x1.79aa65d837b6dp-54}, {0x1.0e3ec32d3d1a2p+0, 0x1.ebe3d702f9cd1p-60},
    {0x1.11301d0125b51p+0, -0x1.556522a2fbd0ep-54}, {0x1.1429aaea92de0p+0, -0x1.1c923b9d5f416p-54},
    {0x1.172b83c7d517bp+0, -0x1.01b15eaa59348p-55}, {0x1.1a35beb6fcb75p+0, 0x1.b898c3f1353bfp-55},
    {0x1.1d4873168b9aap+0, 0x1.aecf73e3a2f60p-54}, {0x1.2063b88628cd6p+0, 0x1.a6f4144a6c38dp-55},
    {0x1.2387a6e756238p+0, 0x1.68efde3a8a894p-54}, {0x1.26b4565e27cddp+0, 0x1.0472b981fe7f2p-55},
    {0x1.29e9df51fdee1p+0, 0x1.2f7e16d09ab31p-55}, {0x1.2d285a6e4030bp+0, 0x1.b3782720c0ab4p-55},
    {0x1.306fe0a31b715p+0, 0x1.34d754db0abb6p-55}, {0x1.33c08b26416ffp+0, 0x1.fdd395dd3f84ap-55},
    {0x1.371a7373aa9cbp+0, -0x1.24aedcc4b5068p-54}, {0x1.3a7db34e59ff7p+0, -0x1.1d1e83e9436d2p-56},
    {0x1.3dea64c123422p+0, 0x1.59f48a72a4c6dp-55}, {0x1.4160a21f72e2ap+0, -0x1.8a78f4817895bp-58},
    {0x1.44e086061892dp+0, 0x1.363ed60c2ac11p-59}, {0x1.486a2b5c13cd0p+0, 0x1.ecce1daa10379p-57},
    {0x1.4bfdad5362a27p+0, 0x1.690cebb7aafb0p-56}, {0x1.4f9b2769d2ca7p+0, -0x1.f94340071a38ep-55},
    {0x1.5342b569d4f82p+0, -0x1.8dec6bd0f385fp-56}, {0x1.56f4736b527dap+0, 0x1.3350518fdd78ep-54},
    {0x1.5ab07dd485429p+0, 0x1.063e1e21c5409p-54}, {0x1.5e76f15ad2148p+0, 0x1.432e62b64c035p-54},
    {0x1.6247eb03a5585p+0, -0x1.c33c53bef4da8p-55}, {0x1.6623882552225p+0, -0x1.3cedd78565858p-54},
    {0x1.6a09e667f3bcdp+0, -0x1.3b3efbf5e2228p-54}, {0x1.6dfb23c651a2fp+0, -0x1.367efb86da9eep-57},
    {0x1.71f75e8ec5f74p+0, -0x1.81f647e5a3ecfp-56}, {0x1.75feb564267c9p+0, -0x1.619321e55e68ap-55},
    {0x1.7a11473eb0187p+0, -0x1.b32dcb94da51dp-56}, {0x1.7e2f336cf4e62p+0, 0x1.5ebe1abd66c55p-57},
    {0x1.82589994cce13p+0, -0x1.369b6f13b3734p-54}, {0x1.868d99b4492edp+0, -0x1.4d450d872576ep-54},
    {0x1.8ace5422aa0dbp+0, 0x1.db72fc1f0eab4p-55}, {0x1.8f1ae99157736p+0, 0x1.bf68359f35f44p-56},
    {0x1.93737b0cdc5e5p+0, -0x1.da9b88b6c1e29p-58}, {0x1.97d829fde4e50p+0, -0x1.2434322f4f9aap-54},
    {0x1.9c49182a3f090p+0, 0x1.1affc2b91ce27p-56}, {0x1.a0c667b5de565p+0, -0x1.7c50422622263p-55},
    {0x1.a5503b23e255dp+0, -0x1.1bbd1d3bcbb15p-54}, {0x1.a9e6b5579fdbfp+0, 0x1.469846e735ab3p-55},
    {0x1.ae89f995ad3adp+0, 0x1.c1a7792cb3387p-55}, {0x1.b33a2b84f15fbp+0, -0x1.5c3d956dcaebap-58},
    {0x1.b7f76f2fb5e47p+0, -0x1.8d6f438ad9334p-57}, {0x1.bcc1e904bc1d2p+0, 0x1.4ffd70a5fddcdp-56},
    {0x1.c199bdd85529cp+0, 0x1.36eae30af0cb3p-56}, {0x1.c67f12e57d14bp+0, 0x1.4e08fd10959acp-55},
    {0x1.cb720dcef9069p+0, 0x1.76b2c6c921968p-57}, {0x1.d072d4a07897cp+0, -0x1.fad5d3ffffa6fp-55},
    {0x1.d5818dcfba487p+0, 0x1.4a385a63d07a7p-56}, {0x1.da9e603db3285p+0, 0x1.e5a50d5c192acp-55},
    {0x1.dfc97337b9b5fp+0, -0x1.2d52107b43e1fp-55}, {0x1.e502ee78b3ff6p+0, 0x1.4b604603a88d3p-56},
    {0x1.ea4afa2a490dap+0, -0x1.ff7128fd391f0p-55}, {0x1.efa1bee615a27p+0, 0x1.ec3bc41aa2008p-55},
    {0x1.f50765b6e4540p+0, 0x1.a64a931d185eep-55}, {0x1.fa7c1819e90d8p+0, 0x1.7893b4d91cd9dp-56}};

struct PlainExp {
  double T, q;             // exp(x) = T (1 + q)
};
__device__ __forceinline__ bool plain_exp_ok(double x) { return (__double2hiint(x) & 0x7fffffff) < 0x40859000; }
__device__ __forceinline__ PlainExp plain_exp_parts(const double2* tab, double x) {
  const double t = fma(x, kInvLn2, 0x1.8p52);            // the integer 64 m + j in the low word
  const int k = __double2loint(t);
  const double n = t - 0x1.8p52;
  const double2 e = tab[k & 63];
  const double h = fma(n, -kLn2Hi, x);                   // r without its rounded part
  const double r = fma(n, -kLn2Lo, h);
  double c = fma(r, 1.0 / 720.0, 1.0 / 120.0);
  c = fma(r, c, 1.0 / 24.0);
  c = fma(r, c, 1.0 / 6.0);
  c = fma(r, c, 0.5);
  return PlainExp{__hiloint2double(__double2hiint(e.x) + ((k >> 6) << 20), __double2loint(e.x)),
                  h + fma(r * r, c, fma(n, -kLn2Lo, e.y))};
}
__device__ __forceinline__ double plain_expm1(const double2* tab, double x) {
  if (!plain_exp_ok(x)) return expm1(x);
  const PlainExp p = plain_exp_parts(tab, x);
  return fma(p.T, p.q, p.T - 1.0);
}
__device__ __forceinline__ double plain_exp(const double2* tab, double x) {
  if (!plain_exp_ok(x)) return exp(x);
  const PlainExp p = plain_exp_parts(tab, x);
  return fma(p.T, p.q, p.T);
}

// What the fluxes through one membrane share (GhkShared with its quotients
// over one reciprocal): e1 = exp(-a1), e2 = e1^2, kr = (a1 / d) / expm1(-a1),
// kr2 = 2 kr / (2 + expm1(-a1)).  The product of the two divisors overflows
// from 9.5 V on, where expm1 itself is finite up to twice that: the reciprocal is
// of expm1 alone there, and e2 infinite, so that divalent fluxes are NaN (as the
// formula's quotient of two infinities).  By selects on the exponent bits: a
// branch with two quotients cost clusters of 43,000 to 55,000 cells 3 to 7 %.
struct PlainShared {
  double e1, e2, kr, kr2;
  __device__ __forceinline__ PlainShared(const double2* tab, double v_nonce, double F_RT, double inv_d) {
    const double a1 = v_nonce * F_RT, em1 = plain_expm1(tab, -a1), u = 2.0 + em1;
    const double p = em1 * u;
    e1 = 1.0 + em1;
    e2 = e1 * e1;
    const bool over = __double2hiint(p) >= 0x7ff00000;      // (NaN too; negative products stay above -1)
    const double g = a1 * inv_d * (1.0 / (over ? em1 : p));
    kr = g * (over ? 1.0 : u);
    kr2 = over ? 0.0 : g + g;
  }
};

// The flux factor of charge code zc for a side A -> B: ghk_flux without Dc,
// from kr = a1 / d / expm1(-a1) and kr2 = 2 kr / (2 + expm1(-a1)).
__device__ __forceinline__ double plain_ghk(int zc, double zval, double v_nonce, double F_RT, double inv_d, double kr,
                                            double kr2, double e1, double e2, double cA, double cB) {
  switch (zc) {
    case 1: return kr * (cB - cA * e1);
    case -1: return kr * (cB * e1 - cA);
    case 2: return kr2 * (cB - cA * e2);
    case -2: return kr2 * (cB * e2 - cA);
    default: {
      const double a = ((zval + kNonce) * v_nonce) * F_RT;
      const double ea = exp(-a), den = -expm1(-a);
      return -(a * inv_d) * ((cB - cA * ea) / den);
    }
  }
}

// The same flux as P - Q cA (factors per cell and ion).
__device__ __forceinline__ void plain_pq(int zc, double zval, double v_nonce, double F_RT, double inv_d, double kr,
                                         double kr2, double e1, double e2, double cB, double& P, double& Q) {
  switch (zc) {
    case 1: P = kr * cB; Q = kr * e1; break;
    case -1: P = (kr * e1) * cB; Q = kr; break;
    case 2: P = kr2 * cB; Q = kr2 * e2; break;
    case -2: P = (kr2 * e2) * cB; Q = kr2; break;
    default: {
      const double a = ((zval + kNonce) * v_nonce) * F_RT;
      const double r = -(a * inv_d) / -expm1(-a);
      P = r * cB;
      Q = r * exp(-a);
    }
  }
}

// w with its sign flipped when s is negative
__device__ __forceinline__ double signed_like(double w, int s) {
  return __hiloint2double(__double2hiint(w) ^ (s & 0x80000000), __double2loint(w));
}

// Sums of eight quantities over the 32 lanes of a warp, every pair of
// neighbouring lanes first (the tree of aligned powers of two): three
// exchange rounds that halve the quantities a lane keeps, then two plain
// ones, nine additions in all.  Lane l returns quantity
// 4 (l & 1) + 2 ((l >> 1) & 1) + ((l >> 2) & 1).
__device__ __forceinline__ double warp_tree8(const double (&a)[8]) {
  const int lane = threadIdx.x & 31;
  double b[4], c[2], d;
  const bool h1 = lane & 1, h2 = lane & 2, h4 = lane & 4;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const double keep = h1 ? a[j + 4] : a[j], send = h1 ? a[j] : a[j + 4];
    b[j] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const double keep = h2 ? b[j + 2] : b[j], send = h2 ? b[j] : b[j + 2];
    c[j] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
  }
  {
    const double keep = h4 ? c[1] : c[0], send = h4 ? c[0] : c[1];
    d = keep + __shfl_xor_sync(0xffffffffu, send, 4);
  }
  d += __shfl_xor_sync(0xffffffffu, d, 8);
  d += __shfl_xor_sync(0xffffffffu, d, 16);
  return d;
}
__device__ __forceinline__ int tree8_ion() {
  const int lane = threadIdx.x & 31;
  return 4 * (lane & 1) + 2 * ((lane >> 1) & 1) + ((lane >> 2) & 1);
}

// rows [0, n) of src ([.][I]), 32 at a time, into dst rows of their sums:
// warps of the CTA in turn.  The caller synchronises.
__device__ __forceinline__ void tree_rows(const double* src, int n, int I, double* dst, int stride_dst) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int c = threadIdx.x >> 5; c * 32 < n; c += nw) {
    double a[8];
    const int r = c * 32 + lane;
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = (i < I && r < n) ? __ldcg(src + (size_t)r * I + i) : 0.0;
    const double s = warp_tree8(a);
    const int i = tree8_ion();
    if (lane < 8 && i < I) dst[(size_t)c * stride_dst + i] = s;
  }
}

// CTAs per SM: four (64 registers) at 100k cells 100.1 us a step against 108.1
// with three (70 registers); extracellular spaces (78 registers) 59.6 us with
// three, 60.6 with four, at 20,400 cells.
template <int ZP, bool GATED, bool RES, bool ECM>
__global__ void __launch_bounds__(kPlainT, RES ? 1 : (ECM ? 3 : 4))
k_plain_step(PlainGeom g, StepPtrs p, StepConst k, PlainRun r, EnvNp en) {
  static_assert(!(RES && ECM), "the grid's own launches separate the steps");
  using IS = PlainIons<ZP>;
  constexpr int T = kPlainT, NI = IS::NI;
  extern __shared__ double sm[];
  __shared__ int s_flag;
  __shared__ double2 stab[64];            // kExpTab
  const int I = IS::n(k);
  const PlainSmem L(r.nc_max, r.ne_max, r.nm_max, I, GATED, ECM);
  double *sQ = sm + L.q, *sv = sm + L.v, *scm = sm + L.cm, *scc = sm + L.cc, *sx = sm + L.x, *s1 = sm + L.s1,
         *sk = sm + L.k, *senv = sm + L.env, *slvl = sm + L.lvl, *sga = sm + L.ga, *sgg = sm + L.gg, *sen = sm + L.en, *spm = sm + L.pm;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, b = blockIdx.x;

  if (t < 64) stab[t] = kExpTab[t];
  // A streaming launch releases the next one as its CTAs exit: released at its
  // start, the next step's CTAs take whatever room the SMs have and the load
  // ends up uneven (20,400 cells 33.2 -> 41.5 us).
  if (!RES) grid_wait();
  if (ECM && b >= g.ntile) {
    env_np_flux<double>(en, (b - g.ntile) * T + t);
    return;   // (an exited CTA has released the next kernel)
  }
  const int2 tl = g.tile[b];
  const int c0 = tl.x, nc = tl.y;
  const int cl = g.tile_cl[b];
  const int m0 = g.cell_ptr[c0], m1 = g.cell_ptr[c0 + nc];
  const int e0 = g.ent_ptr[b], ne = g.ent_ptr[b + 1] - e0, nl = g.n_local[b];
  const double pcoef = p.pump_coef[cl];
  const double *vin = r.vm[0], *cin = r.ccm[0];
  double *vout = r.vm[1], *cout = r.ccm[1];

  // ---- the tile's state
  for (int q = t; q < nc * I; q += T) {
    const int lc = q / I, i = q - lc * I;
    scm[q] = cin[(size_t)i * g.C + c0 + lc];
    scc[q] = p.cc[(size_t)i * g.C + c0 + lc];
  }
  for (int q = t; q < nc; q += T) sv[q] = vin[g.cell_ptr[c0 + q]];
  if (!ECM && t < I) senv[t] = r.cenv[(size_t)cl * I + t];
  for (int q = t; q < 8 * kPlainRows; q += T) slvl[q] = 0.0;
  __syncthreads();

  // junction entry e: Q of every ion from the own side into the partner
  auto entry = [&](int e, bool halo) {
    const int4 en = g.ent[e0 + e];
    const double v1 = sv[en.x] + kNonce;
    const double vn = halo ? __ldcg(vin + en.z) : sv[en.y];
    double cB[NI];
#pragma unroll
    for (int i = 0; i < NI; ++i)
      if (i < I) cB[i] = halo ? __ldcg(cin + (size_t)i * g.C + en.y) : scm[en.y * I + i];
    const double vgj = (vn + kNonce) - v1;        // update_gj, sim.py:2166
    const double vg1 = vgj + kNonce;
    const PlainShared s(stab, vg1, k.F_RT, k.inv_gj_len);
#pragma unroll
    for (int i = 0; i < NI; ++i)
      if (i < I)
        sQ[e * I + i] = plain_ghk(IS::zc(k, i), k.z[i], vg1, k.F_RT, k.inv_gj_len, s.kr, s.kr2, s.e1, s.e2,
                                  scm[en.x * I + i], cB[i]);
    if (GATED) {
      // Gap_Junction.run (channels/gap_junction.py:52-81): one implicit Euler
      // update per ion with these two coefficients (phase G)
      const double V1 = 1.0e3 * fabs(vgj);
      const double al = kGjLambda * plain_exp(stab, -kGjA1 * (V1 - k.gj_vth));
      double be = kGjLambda * plain_exp(stab, kGjA2 * (V1 - k.gj_vth));
      be = be / (1.0 + 50.0 * be);
      sga[2 * e] = k.gj_dt_ms * (al + be * k.gj_min);
      sga[2 * e + 1] = 1.0 / (1.0 + al * k.gj_dt_ms + be * k.gj_dt_ms);
    }
  };
  // cell lc: the shared exponentials of its Vmem
  auto cell_exp = [&](int lc) {
    const PlainShared s(stab, sv[lc] + kNonce, k.F_RT, k.inv_tm);
    double* o = sk + lc * kPlainCell;
    o[PK_K1] = s.kr;
    o[PK_E1] = s.e1;
    o[PK_K2] = s.kr2;
    o[PK_E2] = s.e2;
    o[PK_DTV] = k.dt * g.ivol[c0 + lc];
  };
  // cell lc: its pumps (bit 0 Na/K, bit 1 Ca), times the cell's membrane area
  auto cell_pump = [&](int lc, int which) {
    double* o = sk + lc * kPlainCell;
    const double e1 = o[PK_E1];
    const double* cm = scm + lc * I;
    if (ECM) {
      // pump_fna with the cell's share in PC and PR: PC (k2 - PR nao^3) / (1 +
      // k2), k2 = (ko / KmK)^2 (the quotient's ko^2 cancels against k2)
      const double nai = cm[k.iNa] * 1e-3, ki = cm[k.iK] * 1e-3;
      const double xna = cm[k.iNa] * k.inv_KmNa, c = k.inv_KmK * 1e3;
      const double na3 = xna * xna * xna;
      o[PK_PC] = pcoef * (na3 * k.atp_term) / ((1.0 + na3) * k.atp_den);
      o[PK_PR] = (k.qnum_c * (ki * ki) * e1 * (c * c)) / (k.qden_c * (nai * nai * nai) * k.K0);
      return;
    }
    const double sa = g.sa[c0 + lc];
    if (which & 1) {
      double fna = 0.0;
      if (pcoef != 0.0)                           // Na/K-ATPase (sim.py:1196-1234)
        fna = pump_fna<double>(k, pcoef, e1, cm[k.iNa], senv[k.iNa], cm[k.iK], senv[k.iK]);
      o[PK_FNA] = fna * sa;
    }
    if ((which & 2) && k.iCa >= 0)                // ca_handler (sim.py:2126-2155)
      o[PK_FCA] = pump_fca<double>(k, e1, scc[lc * I + k.iCa], senv[k.iCa]) * sa;
  };

  const int nlp = (nl + 31) & ~31;                // whole warps of local entries, then the cells
  unsigned bad = 0, neg = 0, nanv = 0;
  int step = 0;
  const int n_steps = RES ? r.n_steps : 1;
  for (; step < n_steps; ++step) {
    // ---- A: what needs only the tile
    for (int q = t; q < nlp + nc; q += T) {
      if (q < nlp) {
        if (q < nl) entry(q, false);
      } else {
        cell_exp(q - nlp);
        if (!RES || step == 0) cell_pump(q - nlp, 3);
      }
    }
    if (RES && step > 0) {
      // the other tiles' step: the environment (every CTA adds the same tile
      // parts in the same tree), then the pumps
      if (!res_wait(r.ctl, (unsigned)step * gridDim.x, r.timeout_ns, &s_flag)) break;
      const double* part = r.part + (size_t)(step & 1) * g.ntile * I;
      tree_rows(part, g.ntile, I, slvl, 8);
    }
    for (int q = nl + t; q < ne; q += T) entry(q, true);
    __syncthreads();
    if (RES && step > 0) {
      if (t < I) {
        // kPlainRows rows of 32 tiles (the launch rule)
        const double a = (slvl[t] + slvl[8 + t]) + (slvl[16 + t] + slvl[24 + t]);
        const double c = (slvl[32 + t] + slvl[40 + t]) + (slvl[48 + t] + slvl[56 + t]);
        senv[t] = senv[t] - (a + c) * r.env_scale[cl];
      }
      __syncthreads();
      // (on the step's critical path: the two pumps in different warps; with
      // both in one, a gated step of 2,878 cells took 16.3 us, 15.3 now)
      if (k.iCa < 0) {
        for (int q = t; q < nc; q += T) cell_pump(q, 1);
      } else {
        const int ncp = (nc + 31) & ~31;
        for (int q = t; q < 2 * ncp; q += T) {
          const int lc = q < ncp ? q : q - ncp;
          if (lc < nc) cell_pump(lc, q < ncp ? 1 : 2);
        }
      }
      __syncthreads();
    }
    // ---- M: each membrane's environment and pump
    if (ECM) {
      for (int m = m0 + t; m < m1; m += T) {
        const int ge = g.map_env[m], lc = g.m2c[m] - c0;
        double ce[NI];
#pragma unroll
        for (int i = 0; i < NI; ++i)
          if (i < I) ce[i] = r.cenv[(size_t)i * g.G + ge];
#pragma unroll
        for (int i = 0; i < NI; ++i)
          if (i < I) sen[(m - m0) * I + i] = ce[i];
        double f = 0.0;
        if (pcoef != 0.0) {
          const double cna = r.cenv[(size_t)k.iNa * g.G + ge], cko = r.cenv[(size_t)k.iK * g.G + ge];
          const double* o = sk + lc * kPlainCell;
          const double nao = cna * 1e-3, xk = cko * k.inv_KmK, k2 = xk * xk;
          f = o[PK_PC] * (k2 - o[PK_PR] * (nao * nao * nao)) / (1.0 + k2);
          if ((__double2hiint(f) & 0x7ff00000) == 0x7ff00000 || cko == 0.0)   // a vanishing quotient: the
            f = pump_fna<double>(k, pcoef, o[PK_E1], scm[lc * I + k.iNa], cna, scm[lc * I + k.iK], cko);   // reference's value
        }
        spm[m - m0] = f * g.mem_sa[m];
      }
      __syncthreads();
    }
    // ---- G: the gated open fractions, one lane per membrane
    if (GATED) {
      for (int m = m0 + t; m < m1; m += T) {
        const int e = g.mem_gate[m];
        const double ga = sga[2 * e], gr = sga[2 * e + 1], sa = g.mem_sa[m];
        double gg = p.gjo[m];
        for (int i = 0; i < I; ++i) {
          gg = k.gj_block * ((gg + ga) * gr);
          sgg[(m - m0) * I + i] = gg * sa;
        }
        p.gjo[m] = gg;
      }
      __syncthreads();
    }
    // ---- C: lane per (cell, ion): update_all_concs
    const bool last = step + 1 == n_steps;
    for (int q = t; q < nc * I; q += T) {
      const int lc = q / I, i = q - lc * I, c = c0 + lc;
      const int a0 = g.cell_ptr[c], a1 = g.cell_ptr[c + 1];
      const double* o = sk + lc * kPlainCell;
      double s2 = 0.0, S = 0.0, P = 0.0, Q = 0.0, fp = 0.0;
      if (ECM) {
        plain_pq(IS::zc(k, i), k.z[i], sv[lc] + kNonce, k.F_RT, k.inv_tm, o[PK_K1], o[PK_K2], o[PK_E1], o[PK_E2],
                 scm[q], P, Q);
        fp = i == k.iNa ? 1.0 : i == k.iK ? -(2.0 / 3.0) : 0.0;
      }
      for (int m = a0; m < a1; ++m) {
        if (ECM) {
          const int ml = m - m0;
          const double a = g.dsa[(size_t)m * I + i] * (P - Q * sen[ml * I + i]) + fp * spm[ml];
          p.mem_flux_sa[(size_t)g.env_slot[m] * kMfs + i] = a;
          S += a;
        }
        const int me = g.mem_ent[m];
        if (me == kPlainNone) continue;
        const double w = GATED ? sgg[(m - m0) * I + i] : g.mem_w[m];
        s2 += signed_like(w, ~me) * sQ[(me >= 0 ? me : ~me) * I + i];   // -w on the own side
      }
      if (!ECM) {
        S = g.dsa[(size_t)i * g.C + c] * plain_ghk(IS::zc(k, i), k.z[i], sv[lc] + kNonce, k.F_RT, k.inv_tm, o[PK_K1],
                                                 o[PK_K2], o[PK_E1], o[PK_E2], senv[i], scm[q]);
        if (i == k.iNa) S = o[PK_FNA] + S;
        else if (i == k.iK) S = -(2.0 / 3.0) * o[PK_FNA] + S;
        if (i == k.iCa) S = S + o[PK_FCA];
      }
      s1[q] = S;
      double x = scc[q] + S * o[PK_DTV];              // update_Co, sim_toolbox.py:1182-1183
      sx[q] = x;
      cout[(size_t)i * g.C + c] = x;        // cc_at_mem = cX_cell[mem_to_cells]
      const double dg = GATED ? k.dgj_gs[i] : k.dgj_gs[i] * k.gj_block;
      x = x + (dg * s2) * o[PK_DTV];                  // gap-junction term, sim.py:2105-2108
      const int hx = __double2hiint(x);               // integer tests: no FP64 pipe
      const bool nan = (hx & 0x7fffffff) > 0x7ff00000 || ((hx & 0x7fffffff) == 0x7ff00000 && __double2loint(x));
      bad += nan;
      if (hx < 0 && !nan && ((hx & 0x7fffffff) | __double2loint(x))) { x = 0.0; ++neg; }   // no_negs
      scc[q] = x;
      if (last) p.cc[(size_t)i * g.C + c] = x;
    }
    __syncthreads();
    // ---- D: Vmem (the last warps) and the tile's part of the environment
    for (int lc = T - 1 - t; lc < nc; lc += T) {
      double rho = 0.0;                               // rho_cells, ion_current.py:19
#pragma unroll
      for (int i = 0; i < NI; ++i)
        if (i < I) rho += k.zF[i] * scc[lc * I + i];
      const double v = k.inv_cm * (rho * g.diviterm[c0 + lc]);   // sim.py:2027-2029
      sv[lc] = v;
      const int a0 = g.cell_ptr[c0 + lc];
      if (v != v) nanv += g.cell_ptr[c0 + lc + 1] - a0;
      if (RES) vout[a0] = v;                 // what the other tiles read
    }
    if (!ECM) {
      // lane l: cells [l, l + 1), or a run of 2 or 4, pairs first
      double* part = r.part + (RES ? (size_t)((step + 1) & 1) * g.ntile * I : (size_t)0);
      for (int i = warp; i < I; i += T / 32) {
        double a;
        auto at = [&](int lc) { return lc < nc ? s1[lc * I + i] : 0.0; };
        if (r.nc_max <= 32) a = at(lane);
        else if (r.nc_max <= 64) a = at(2 * lane) + at(2 * lane + 1);
        else a = (at(4 * lane) + at(4 * lane + 1)) + (at(4 * lane + 2) + at(4 * lane + 3));
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (lane == 0) part[(size_t)b * I + i] = a;
      }
    }
    if (RES) {
      for (int q = t; q < nc * I; q += T) scm[q] = sx[q];
      double* w = vout; vout = const_cast<double*>(vin); vin = w;
      w = cout; cout = const_cast<double*>(cin); cin = w;
      __syncthreads();
      if (t == 0) res_arrive(r.ctl);         // a release: the CTA's writes, ordered by the bar.sync, with it
    }
  }
  if (bad) atomicAdd(&p.status[1], (unsigned long long)bad);
  if (neg) atomicAdd(&p.status[2], (unsigned long long)neg);
  if (nanv) atomicAdd(&p.status[0], (unsigned long long)nanv);

  if (RES) {
    if (step < n_steps) return;                       // the barrier gave up
    // Vmem of every membrane, and the environment of the last step (CTA 0)
    double* vfin = const_cast<double*>(vin);
    for (int m = m0 + t; m < m1; m += T) vfin[m] = sv[g.m2c[m] - c0];
    if (b == 0) {
      if (!res_wait(r.ctl, (unsigned)step * gridDim.x, r.timeout_ns, &s_flag)) return;
      tree_rows(r.part + (size_t)(step & 1) * g.ntile * I, g.ntile, I, slvl, 8);
      __syncthreads();
      if (t < I) {
        const double a = (slvl[t] + slvl[8 + t]) + (slvl[16 + t] + slvl[24 + t]);
        const double c = (slvl[32 + t] + slvl[40 + t]) + (slvl[48 + t] + slvl[56 + t]);
        r.cenv[t] = senv[t] - (a + c) * r.env_scale[0];
      }
    }
    return;
  }

  // ---- streaming: Vmem of every membrane, then the environment by tickets
  __syncthreads();
  for (int m = m0 + t; m < m1; m += T) vout[m] = sv[g.m2c[m] - c0];
  if (ECM) {
    grid_release();
    return;
  }
  const int ct0 = g.cl_tile[cl], nt = g.cl_tile[cl + 1] - ct0;
  const int grp = (b - ct0) >> 5, ngrp = (nt + 31) >> 5;
  const int g0 = g.cl_group[cl];
  unsigned* tk = r.ticket + g0 + cl;                  // the cluster's groups, then its own counter
  if (t == 0) {
    __threadfence();
    const unsigned n = (unsigned)min(32, nt - 32 * grp);
    s_flag = atomicAdd(&tk[grp], 1u) == n - 1u;
  }
  __syncthreads();
  if (!s_flag) return;
  __threadfence();
  // rows of parts, level by level: 32 tiles -> group -> 32 groups -> ...
  double* lv = r.gpart + (size_t)(2 * g0 + 8 * cl) * I;
  {
    const double* src = r.part + (size_t)(ct0 + 32 * grp) * I;
    if (warp == 0) {
      double a[8];
      const int n = min(32, nt - 32 * grp);
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = (i < I && lane < n) ? __ldcg(src + (size_t)lane * I + i) : 0.0;
      const double s = warp_tree8(a);
      const int i = tree8_ion();
      if (lane < 8 && i < I) lv[(size_t)grp * I + i] = s;
    }
  }
  __syncthreads();
  if (t == 0) {
    tk[grp] = 0u;
    __threadfence();
    s_flag = atomicAdd(&tk[ngrp], 1u) == (unsigned)ngrp - 1u;
  }
  __syncthreads();
  if (!s_flag) return;
  __threadfence();
  int n = ngrp;
  while (n > 1) {
    double* up = lv + (size_t)n * I;
    tree_rows(lv, n, I, up, I);
    __threadfence_block();
    __syncthreads();
    lv = up;
    n = (n + 31) >> 5;
  }
  if (t < I) {
    double* ce = r.cenv + (size_t)cl * I + t;
    *ce = *ce - __ldcg(lv + t) * r.env_scale[cl];     // sim_toolbox.py:1196-1205
  }
  if (t == 0) tk[ngrp] = 0u;
}

// sum of Dm_i * mem_sa over the cell's membranes, lane per (ion, cell)
static __global__ void k_plain_dsa(int C, int M, int I, const int* __restrict__ cell_ptr,
                                   const double* __restrict__ Dm, const double* __restrict__ mem_sa, double* dsa) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (c >= C) return;
  double s = 0.0;
  for (int m = cell_ptr[c]; m < cell_ptr[c + 1]; ++m) s += Dm[(size_t)i * M + m] * mem_sa[m];
  dsa[(size_t)i * C + c] = s;
}

// the membranes' junction weights times area, the cells' areas and 1 / cell_vol
static __global__ void k_plain_static(int C, const int* __restrict__ cell_ptr, const double* __restrict__ gj_w,
                                      const double* __restrict__ mem_sa, const double* __restrict__ cell_vol,
                                      double* mem_w, double* sa, double* ivol) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  double s = 0.0;
  for (int m = cell_ptr[c]; m < cell_ptr[c + 1]; ++m) {
    mem_w[m] = gj_w[m] * mem_sa[m];
    s += mem_sa[m];
  }
  sa[c] = s;
  ivol[c] = 1.0 / cell_vol[c];
}

// Dm_i * mem_sa of every membrane, ion contiguous (ECM)
static __global__ void k_plain_dsam(int M, int I, const double* __restrict__ Dm, const double* __restrict__ mem_sa,
                                    double* dsam) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= M) return;
  for (int i = 0; i < I; ++i) dsam[(size_t)m * I + i] = Dm[(size_t)i * M + m] * mem_sa[m];
}

// launchers (bx_step_f64_small.cu); ecm: with the grid's flux in en.nblk more blocks
cudaError_t launch_plain_step(bool six, bool gated, bool ecm, cudaStream_t s, const PlainGeom& g, const StepPtrs& p,
                              const StepConst& k, const PlainRun& r, const EnvNp& en);
// counter: the byte the barrier's counter is filled with (0; kStuckByte: a count
// that no wait of this launch can reach)
constexpr int kStuckByte = 0x80;
cudaError_t launch_plain_resident(bool six, bool gated, cudaStream_t s, const PlainGeom& g, const StepPtrs& p,
                                  const StepConst& k, const PlainRun& r, int counter);
// CTAs of the resident form that fit one SM with this much shared memory (0: none)
cudaError_t plain_resident_per_sm(bool six, bool gated, size_t smem, int* per_sm);
// the shared-memory limit of both forms, raised once per device
cudaError_t plain_smem_attr(bool six, bool gated, bool ecm, size_t smem);

}  // namespace bx
