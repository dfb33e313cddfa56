// Spin-temperature step (_ComputeTs, src/core/ComputeTs.c:85-1554) on sm_100a, with the AGN
// X-ray channels (Flag_IncludeAGNXray) and without the mini-halo channels.
//
// Inhomogeneous branch, per snapshot:
//   1. FP64 reductions of the collapse fraction and <x_e> (ComputeTs.c:585-677)
//   2. frequency-integral tables on a side stream (rg_freq.cu); host: Lyman-n sums, prefactors
//   3. forward r2c of every source grid (this snapshot's sfr / xray_luminosity and the
//      history slots the shells use); each shell's source is a linear combination of them
//      (the history re-weighting of :366-478), formed in k-space on load
//   4. shells in batches: x pass (combination, TsHeatingFilterType window), y pass, z pass
//      that turns the grids of every shell (sfr, X-ray, then the AGN soft and / or hard
//      emissivity) into the four per-cell sums of
//      evolveInt (X-ray heating, ionisation and Lyman-alpha integrands, stellar Lyman-alpha)
//      without storing the reference's SMOOTHED_*[nS N^3] arrays.
//      The X-ray sums are linear in the filtered X-ray grids (they are not clamped) and piecewise
//      linear in the cell's x_e, so with x_e on few table nodes they are formed in k-space, one
//      field per node and kind (k_ts_nodes), instead of one X-ray transform per shell.
//      With the sharp-k window the modes beyond a shell's cut are zero: the x pass skips their
//      columns, the y pass their lines, and the z pass does not read their planes.
//   5. per cell, FP64: evolveInt, the Euler step of x_e and T_K, get_Ts, and the FP64 sums
// Homogeneous branch (zp >= ReionMaxHeatingRedshift): RECFAST x_e and T_K, get_Ts with no
// Lyman-alpha coupling (:252-331).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "rg_freq.h"
#include "rg_internal.h"
#include "rg_pass.cuh"
#include "rg_tma.cuh"
#include "rg_xphys.h"
#include "rg_xray.h"

namespace rg {

constexpr int TS_KB = 8;        // spare slots for combinations, and the least shells per batch
constexpr int TS_MAXB = 40;     // most shells per batch
constexpr int TS_MAXSRC = 4;    // sources combined into one shell
constexpr int TS_NSUM = 9;      // evolve sums (7, 8: the AGN heating of the two AGN units)
constexpr int KSPL = 27;        // knots of the largest kappa table

constexpr int KLUT = 64;
struct KappaSpline {
  int n;
  int lut[KLUT];           // last knot at or below the start of each of KLUT equal steps of the table
  double x0, inv_step;
  double x[KSPL], y[KSPL], b[KSPL], c[KSPL], d[KSPL];
};

// per-snapshot constants of the per-cell physics (the factors of xcoll, taugp, xalpha_tilde,
// dT_comp and evolveInt that depend on the redshift only), computed on the host in FP64
struct TsZConst {
  double Trad, inv_Trad;       // TCMB (1 + z), z the float redshift
  double xc_H, xc_e, xc_p;     // T21 / Trad / A10 x {No, N_b0, No} (1 + z)^3   (xcoll_HI/elec/prot)
  double tgp0;                 // 1.342881e-7 / hubble(z) No (1 + z)^3          (taugp)
  double xa0;                  // 1.66e11 / (1 + z)                             (xalpha_tilde)
  double nb0;                  // N_b0 (1 + z)^3                                (evolveInt n_b)
  double comp0;                // -1.51e-4 / (H(z) / H0) / h Trad^4 / (1 + z)    (dT_comp)
  double dadia0;               // 3 / (1 + z)
  double f_H, f_He;
};

struct TsDev {
  KappaSpline k10, kel, kpH;
};
// the scalars travel as a kernel parameter (operands of the constant bank)
struct TsPar {
  TsZConst z;
  int max_iter;   // get_Ts fixed-point iterations before a cell counts as not converged
};

__device__ __forceinline__ double spline_eval(const KappaSpline& s, double x) {
  // the last knot at or below x (x lies in the table), from the step's first candidate
  int lo = s.lut[min(max((int)((x - s.x0) * s.inv_step), 0), KLUT - 1)];
  while (lo < s.n - 2 && !(s.x[lo + 1] > x)) ++lo;
  const double dx = x - s.x[lo];
  return s.y[lo] + dx * (s.b[lo] + dx * (s.c[lo] + dx * s.d[lo]));
}

// log kappa_10 at log T (XRayHeatingFunctions.c:1728-1822): below the table its first value,
// above it the T^0.381 power law log(exp(y_n) (T / exp(x_n))^0.381) = y_n + 0.381 (log T - x_n)
__device__ __forceinline__ double log_kappa_10(const KappaSpline& s, double lt) {
  if (lt < s.x[0]) return s.y[0];
  if (lt > s.x[s.n - 1]) return s.y[s.n - 1] + 0.381 * (lt - s.x[s.n - 1]);
  return spline_eval(s, lt);
}

// log kappa_10_elec / kappa_10_pH at log T (XRayHeatingFunctions.c:1827-1966): linear
// extrapolation of the last segment above the table
__device__ __forceinline__ double log_kappa_table(const KappaSpline& s, double lt) {
  if (lt < s.x[0]) return s.y[0];
  if (lt > s.x[s.n - 1])
    return s.y[s.n - 1] + ((s.y[s.n - 1] - s.y[s.n - 2]) / (s.x[s.n - 1] - s.x[s.n - 2]) * (lt - s.x[s.n - 1]));
  return spline_eval(s, lt);
}

// get_Ts with xcoll and the Wouthuysen-Field coupling (XRayHeatingFunctions.c:1639-1726,
// 1973-2008).  The factors that do not change across the fixed-point iterations (xcoll, the
// S_alpha terms in T_K only, xi) are evaluated once per cell.  The loop is capped at
// P.max_iter iterations (10000 unless a test lowers it); a cell that reaches the cap counts in
// *nonconv.
// The iteration runs on u = 1 / T_S, one division a step; |T_S - T_S,old| / T_S = |u_old - u| / u_old.
__device__ __forceinline__ float get_Ts(const TsDev& C, const TsPar& P, float delta, float TK, float xe, float Jalpha,
                                        float* curr_xalpha, int* nonconv) {
  const TsZConst& Z = P.z;
  const double tk = (double)TK, d1 = 1.0 + (double)delta, x = (double)xe;
  const double lt = log(tk);
  const double xc = Z.xc_H * (1.0 - x) * d1 * exp(log_kappa_10(C.k10, lt)) +
                    Z.xc_e * x * d1 * exp(log_kappa_table(C.kel, lt)) +
                    Z.xc_p * x * d1 * exp(log_kappa_table(C.kpH, lt));
  const double itk = 1.0 / tk;
  double TS;
  if ((double)Jalpha > 1.0e-20) {
    const double tgp = Z.tgp0 * d1 * (1.0 - x);
    const double xi = cbrt(1.0e-7 * tgp * itk * itk);
    const double den = 1.0 + 2.98394 * xi + 1.53583 * xi * xi + 3.85289 * xi * xi * xi;
    const double sa = 1.0 - 0.0631789 * itk + 0.115995 * itk * itk;    // S_alpha terms in T_K only
    const double sb = (-0.401403 + 0.336463 * itk) * itk;                 // times 1 / T_S
    const double xaj = Z.xa0 * (double)Jalpha / den;
    const double ctc = 0.405535 * itk;
    const double den_c = Z.inv_Trad + xc * itk, num_c = 1.0 + xc, tce_c = itk - ctc * itk;
    double u = Z.inv_Trad, xa_tilde = 0.0;
    int it = 0;
    for (;;) {
      if (++it > P.max_iter) {
        *nonconv += 1;
        break;
      }
      const double uold = u;
      xa_tilde = xaj * (sa + sb * u);
      // 1 / Tc_eff = 1 / T_K + ctc (1 / T_S - 1 / T_K)
      u = (den_c + xa_tilde * (tce_c + ctc * u)) / (num_c + xa_tilde);
      if (!(u > 0.0 && fabs(uold - u) > 1.0e-3 * uold)) break;
    }
    TS = 1.0 / u;
    *curr_xalpha = (float)xa_tilde;
  } else {
    TS = (1.0 + xc) / (Z.inv_Trad + xc * itk);
    *curr_xalpha = 0;
  }
  if (TS < 0.) TS = fabs(TS);
  return (float)TS;
}

// alpha_A (XRayHeatingFunctions.c:1576-1584): exp of a degree-9 polynomial in
// log(T / 1.1604505e4), evaluated by Horner's rule
__device__ __forceinline__ double alpha_A(double T) {
  const double l = log(T / 1.1604505e4);
  const double poly =
      -28.6130338 +
      l * (-0.72411256 +
           l * (-2.02604473e-2 +
                l * (-2.38086188e-3 +
                     l * (-3.21260521e-4 +
                          l * (-1.42150291e-5 +
                               l * (4.98910892e-6 + l * (5.75561414e-7 + l * (-1.85676704e-8 + l * -3.07113524e-9))))))));
  return exp(poly);
}

// ---------------------------------------------------------------------------
// block sums (deterministic) -> partials[block][K]

template <int K>
__device__ __forceinline__ void block_sum_dyn(double (&acc)[K], double* out) {
  __shared__ double s_red[32][K];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < K; ++i) {
    double v = acc[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) s_red[wid][i] = v;
  }
  __syncthreads();
  if (threadIdx.x < K) {
    double v = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += s_red[w][threadIdx.x];
    out[threadIdx.x] = v;
  }
}

// floats as unsigned integers of the same order (and back, on the host)
__device__ __forceinline__ unsigned float_order(float v) {
  const unsigned b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
static float float_of_order(unsigned o) {
  const unsigned b = (o & 0x80000000u) ? (o & 0x7fffffffu) : ~o;
  float v;
  std::memcpy(&v, &b, sizeof(v));
  return v;
}

// What a snapshot's kernels report next to their sums, all zero before the first of them: one memset and no
// copy of its own (it lies behind the sums, d_sums[TS_STATUS]).  As three words set and fetched each by
// itself a homogeneous call took 119 us at 64^3; so it takes 110.
struct TsStatus {
  unsigned xe_top;       // the largest x_e in float_order
  unsigned xe_bottom;    // the smallest, complemented
  int nonconv;           // cells whose get_Ts ran out of iterations
  int pad;
};
constexpr int TS_STATUS = 48;
static_assert(sizeof(TsStatus) == 2 * sizeof(double), "two slots of the sums");

// collapse fraction, <x_e> and the range of x_e over the box (ComputeTs.c:585-677)
__global__ void __launch_bounds__(256) k_ts_reduce0(const float* __restrict__ stars, const float* __restrict__ deltax,
                                                    const float* __restrict__ xe, int n, double Mh2,
                                                    double fourthirds_pi_R3_over_pv, double* partials,
                                                    TsStatus* __restrict__ status) {
  constexpr int U = 4;   // cells of a thread whose loads are in flight together
  const size_t n3 = (size_t)n * n * n, step = (size_t)gridDim.x * 256;
  const double f = fourthirds_pi_R3_over_pv / Mh2;
  double acc[2] = {0.0, 0.0};
  float mn = INFINITY, mx = -INFINITY;
  bool nan = false;
  for (size_t i0 = (size_t)blockIdx.x * 256 + threadIdx.x; i0 < n3; i0 += U * step) {
    float st[U], dx[U], v[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const size_t i = i0 + k * step;
      if (i >= n3) break;
      const size_t ip = i + ((unsigned)i / (unsigned)n) * 2;   // rows of n + 2 values
      st[k] = stars[ip];
      dx[k] = deltax[ip];
      v[k] = xe[ip];
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      if (i0 + k * step >= n3) break;
      const double c = (double)st[k] * f / (1.0 + (double)dx[k]);
      acc[0] += c > 1.0 ? 1.0 : c;
      acc[1] += (double)v[k];
      mn = fminf(mn, v[k]);
      mx = fmaxf(mx, v[k]);
      nan |= v[k] != v[k];
    }
  }
  // the range of x_e as ordered integers; a NaN, which the minimum and maximum pass over, is its top
  unsigned bottom = ~float_order(mn), top = nan ? ~0u : float_order(mx);
  block_sum_dyn<2>(acc, partials + (size_t)blockIdx.x * 2);
  __shared__ unsigned s_bottom, s_top;
  if (threadIdx.x == 0) s_bottom = s_top = 0u;
  __syncthreads();
  bottom = __reduce_max_sync(0xffffffffu, bottom);
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&s_bottom, bottom);
    atomicMax(&s_top, top);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicMax(&status->xe_bottom, s_bottom);
    atomicMax(&status->xe_top, s_top);
  }
}

// ---------------------------------------------------------------------------
// shell x pass: output (r, g) = sum_i cs[r][i] spec[ks[r][i]][g] x window_r, transformed along x

struct TsBatch {
  int nr;
  int chunk;          // shells a block of the x pass takes
  int nk[TS_MAXB];
  int ks[TS_MAXB][TS_MAXSRC];
  float cs[TS_MAXB][TS_MAXSRC];
  int filtered[TS_MAXB];
  int wrow[TS_MAXB];
  int cut[TS_MAXB];     // last n2 that the shell's window keeps (TS_NOCUT: all)
  int gs;             // grids per source: sfr, X-ray, then 0 to 2 AGN bands
  int ng;             // grids per shell: the same, without X-ray where that goes by nodes
  int skip;           // 1: X-ray goes by nodes
};
constexpr int TS_NOCUT = 0x7fffffff;

// Columns beyond a shell's cut hold zeros, which the y pass knows: they are neither read nor written.
// At 512^3 with 40 sharp-k shells the shells' volumes add up to 4 grids of 40 and their columns to 6.
template <int N>
__global__ void __launch_bounds__(Cfg<N>::T* Cfg<N>::BX, (x_pass_minb<N>()))
    k_ts_x(const cf* __restrict__ spec, size_t stride, cf* __restrict__ work, const __grid_constant__ TsBatch bt,
           const float* __restrict__ wtab, int wpitch, const cf* __restrict__ g_tw) {
  constexpr int T = Cfg<N>::T, B = Cfg<N>::BX, V = Cfg<N>::V;
  extern __shared__ cf smem[];
  cf* s_tw = smem;
  cf* xbuf = smem + N;
  const int kz = blockIdx.y;
  const int b = threadIdx.x % B, t = threadIdx.x / B;
  const int y = blockIdx.x * B + b;
  const size_t col = (size_t)kz * N * N + y;
  // the least n2 of the block's columns (|ny| is least at one of its ends)
  const int ya = blockIdx.x * B, yb = ya + B - 1;
  const int na = ya > N / 2 ? N - ya : ya, nb = yb > N / 2 ? N - yb : yb;
  const int n2min = kz * kz + min(na, nb) * min(na, nb);
  load_twiddles<N>(s_tw, g_tw);
  int n2[V];
  const int ny = y > N / 2 ? y - N : y;
#pragma unroll
  for (int sl = 0; sl < V; ++sl) {
    const int p = stage0_pos<N>(t, sl);
    const int nx = p > N / 2 ? p - N : p;
    n2[sl] = nx * nx + ny * ny + kz * kz;
  }
  __syncthreads();
  const int r_end = min(bt.nr, ((int)blockIdx.z + 1) * bt.chunk);
  for (int r = blockIdx.z * bt.chunk; r < r_end; ++r) {
    const int cut = bt.cut[r];
    if (n2min > cut) continue;
    float wv[V];
    if (!bt.filtered[r] || cut != TS_NOCUT) {
#pragma unroll
      for (int sl = 0; sl < V; ++sl) wv[sl] = 1.f;   // sharp-k: the modes beyond the cut are not loaded
    } else {
      const float* wr = wtab + (size_t)bt.wrow[r] * wpitch;
#pragma unroll
      for (int sl = 0; sl < V; ++sl) wv[sl] = __ldg(wr + n2[sl]);
    }
    const int nk = bt.nk[r];
    for (int g = 0; g < bt.ng; ++g) {
      const int gsrc = g > 0 ? g + bt.skip : 0;
      cf* dst = work + ((size_t)r * bt.ng + g) * stride;
      // the combination sum_i c_i spec_i of this thread's V input positions, source by source:
      // the V loads of a source are independent and in flight together (per element the same
      // fmaf sequence in the order of i)
      cf in[V];
#pragma unroll
      for (int sl = 0; sl < V; ++sl) in[sl] = cf{0.f, 0.f};
      for (int i = 0; i < nk; ++i) {
        const float c = bt.cs[r][i];
        const cf* src = spec + ((size_t)bt.ks[r][i] * bt.gs + gsrc) * stride + col;
        cf v[V];
#pragma unroll
        for (int sl = 0; sl < V; ++sl)
          v[sl] = n2[sl] <= cut ? src[(size_t)stage0_pos<N>(t, sl) * N] : cf{0.f, 0.f};
#pragma unroll
        for (int sl = 0; sl < V; ++sl) {
          in[sl].x = fmaf(c, v[sl].x, in[sl].x);
          in[sl].y = fmaf(c, v[sl].y, in[sl].y);
        }
      }
      line_fft<N, true>(
          t, xbuf, s_tw, [&](int, int sl) { return cf{in[sl].x * wv[sl], in[sl].y * wv[sl]}; },
          [&](int p) { return line_addr<N, B>(p, b); }, [&](int p, cf v) { dst[col + (size_t)p * N] = v; });
    }
  }
}

// shell y pass, in place: the columns beyond the cut are zero (the x pass left them unwritten), the
// planes beyond it are not transformed (the z pass does not read them); gridDim.y covers the
// batch's planes.  blockIdx.z: shell r, grid g at work + (r ng + g) stride.
template <int N>
__global__ void __launch_bounds__(YCfg<N>::NTH, RG_MINB(YCfg<N>::NTH))
    k_ts_y(cf* __restrict__ work, size_t stride, const __grid_constant__ TsBatch bt, const cf* __restrict__ g_tw) {
  using Y = YCfg<N>;
  using PL = typename Y::PL;
  constexpr int T = Y::T, B = Y::BY;
  extern __shared__ cf smem[];
  cf* s_tw = smem;
  cf* xbuf = smem + N;
  const int kz = blockIdx.y;
  const int left = bt.cut[blockIdx.z / bt.ng] - kz * kz;   // ny^2 up to this
  if (left < 0) return;
  const int t = threadIdx.x % T, b = threadIdx.x / T;
  load_twiddles_p<PL>(s_tw, g_tw);
  __syncthreads();
  cf* line = work + blockIdx.z * stride + ((size_t)kz * N + blockIdx.x * B + b) * N;
  line_fft_p<PL, true, true>(
      t, xbuf, s_tw,
      [&](int p, int) {
        const int ny = p > N / 2 ? N - p : p;
        return ny * ny <= left ? line[p] : cf{0.f, 0.f};
      },
      [&](int p) { return pos_addr<N>(b, p); }, [&](int p, cf v, int) { line[p] = v; });
}

// ---------------------------------------------------------------------------
// X-ray by nodes: the cell's heating, ionisation and Lyman-alpha sums
//   sum_r xray_r(cell) (P_rk[lo] + (x_e - X[lo]) Q_rk[lo])
// are linear in the filtered grids xray_r and, between the table's x_e nodes X[m], linear in x_e:
//   (1 - t) F_k[lo] + t F_k[lo + 1],  F_k[m] = sum_r f_rk(X[m]) xray_r,  t = (x_e - X[lo]) / (X[lo + 1] - X[lo])
// so the sum over shells is taken in k-space, once per node that the box uses.  3 M transforms
// instead of nS (M nodes: two where the whole box lies between neighbouring nodes); ts_snapshot chooses
// by cost.  At 128^3, 4 nodes and 40 sharp-k shells the X-ray part takes 0.53 ms by nodes, 0.61 by shells.

// Nodes that one chunk of k_ts_nodes (a blockIdx.y) takes: all of them up to 4, else as even as 3 or 4
// nodes a chunk go.
constexpr int ts_node_chunk(int nm) {
  return nm <= 2 ? 2 : (nm == 3 || nm == 5 || nm == 6 || nm == 9) ? 3 : 4;
}
constexpr int ts_node_chunks(int nm) { return (nm + ts_node_chunk(nm) - 1) / ts_node_chunk(nm); }
// Coefficients a launch reads of each shell: those of whole chunks, so up to 2 nodes beyond nm (zeros)
constexpr int ts_node_reads(int nm) { return 3 * ts_node_chunk(nm) * ts_node_chunks(nm); }
constexpr int ts_node_most_reads() {
  int most = 0;
  for (int nm = 1; nm <= x_int_NXHII; ++nm) most = ts_node_reads(nm) > most ? ts_node_reads(nm) : most;
  return most;
}

struct TsNodeShell {
  int nk;                    // sources of the shell
  int filtered, cut;         // as in TsBatch
  int ks[TS_MAXSRC];
  float cs[TS_MAXSRC];
  float f[ts_node_most_reads()];   // coefficient of field 3 j + kind, node m0 + j; zero beyond the last node
};

// fields [f0, f0 + NF) of nf (f0 = blockIdx.y NF): work[f] = sum_r f_r W_r sum_i c_i spec[k_i][1].
// One mode a thread; the shells' coefficients are the same for the whole block (read through L1),
// as are mostly the shells that a warp's modes pass.
template <int NF>
__global__ void __launch_bounds__(256) k_ts_nodes(const cf* __restrict__ spec, size_t stride, int gs,
                                                  cf* __restrict__ work, const TsNodeShell* __restrict__ shells, int nS,
                                                  int nf, const float* __restrict__ wtab, int wpitch, int log2n) {
  const int n = 1 << log2n, f0 = blockIdx.y * NF;
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < stride; i += (size_t)gridDim.x * 256) {
    const int y = (int)(i & (n - 1)), x = (int)((i >> log2n) & (n - 1)), kz = (int)(i >> (2 * log2n));
    const int ny = y > n / 2 ? y - n : y, nx = x > n / 2 ? x - n : x;
    const int n2 = nx * nx + ny * ny + kz * kz;
    cf acc[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) acc[f] = cf{0.f, 0.f};
    for (int r = 0; r < nS; ++r) {
      const TsNodeShell& s = shells[r];
      const int cut = s.cut;
      if (n2 > cut) continue;
      cf v{0.f, 0.f};
      const int nk = s.nk;
      for (int j = 0; j < nk; ++j) {
        const float2 a = __ldg(reinterpret_cast<const float2*>(spec + ((size_t)s.ks[j] * gs + 1) * stride + i));
        v.x = fmaf(s.cs[j], a.x, v.x);
        v.y = fmaf(s.cs[j], a.y, v.y);
      }
      if (s.filtered && cut == TS_NOCUT) {
        const float w = __ldg(wtab + (size_t)r * wpitch + n2);
        v.x *= w;
        v.y *= w;
      }
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        const float c = s.f[f0 + f];
        acc[f].x = fmaf(c, v.x, acc[f].x);
        acc[f].y = fmaf(c, v.y, acc[f].y);
      }
    }
#pragma unroll
    for (int f = 0; f < NF; ++f)
      if (f0 + f < nf) work[(size_t)(f0 + f) * stride + i] = acc[f];
  }
}

// ---------------------------------------------------------------------------
// per-cell evolution (evolveInt + the Euler step + get_Ts, ComputeTs.c:1171-1407)

struct TsEvolve {
  double zp, dzp, dt_dzp, growth, dgrowth, const_zp, conv_star;
  double heat_conv;            // dt_dzp 2 / 3 / k_B
  int no_light;
};

// One cell: sums[0..3] = the four evolveInt shell sums (heat, ion, lya, stellar lya) before
// their snapshot prefactors; updates x_e and T_K, returns T_S and adds the cell to acc[0..6].
__device__ __forceinline__ void evolve_cell(const TsDev& C, const TsPar& P, const TsEvolve& e, float delta, float xef, float tk0,
                                            const double (&sums)[4], float* xn_out, float* tk_out, float* ts_out,
                                            double (&acc)[TS_NSUM], int* nc) {
  const TsZConst& Z = P.z;
  const double x_e = (double)xef, T = (double)tk0;
  const double n_b = Z.nb0 * (double)(1.0f + delta);
  double dxheat_dt = 0, dxion_src = 0, dxlya = 0, dstarlya = 0;
  if (!e.no_light) {
    dxheat_dt = sums[0] * e.const_zp;
    dxion_src = sums[1] * e.const_zp;
    dxlya = sums[2] * (e.const_zp * n_b);
    dstarlya = sums[3] * e.conv_star;
  }
  const double inv1x = 1.0 / (1.0 + x_e);
  const double dxion_sink = alpha_A(T) * CLUMPING_FACTOR * x_e * x_e * Z.f_H * n_b;
  const double dxe_dzp = e.dt_dzp * (dxion_src - dxion_sink);
  double dadia = Z.dadia0;
  if (fabs((double)delta) > FRACT_FLOAT_ERR) {
    const double dl = (double)delta;
    dadia += e.dgrowth * dl / (1.0 + e.growth * dl);      // dgrowth / (1 / delta + growth)
  }
  dadia *= (2.0 / 3.0) * T;
  const double dspec = -dxe_dzp * T * inv1x;
  const double dcomp = Z.comp0 * (x_e / (1.0 + x_e + Z.f_He)) * (Z.Trad - T);
  const double dxheat_dzp = dxheat_dt * e.heat_conv * inv1x;
  const double d1 = dxheat_dzp + dcomp + dspec + dadia;
  const double d2 = dxlya + dstarlya;
  const double d4 = e.dt_dzp * dxion_src;
  float xn = (float)((double)xef + dxe_dzp * e.dzp);
  if (xn > 1)
    xn = (float)(1 - FRACT_FLOAT_ERR);
  else if (xn < 0)
    xn = 0;
  float tk = tk0;
  if (tk < MAX_TK) tk = (float)((double)tk + d1 * e.dzp);
  if (tk < MIN_TK) tk = (float)(TCMB * (1 + e.zp));
  float xa;
  const float ts = get_Ts(C, P, delta, tk, xn, (float)d2, &xa, nc);
  *xn_out = xn;
  *tk_out = tk;
  *ts_out = ts;
  acc[0] += d2;
  acc[1] += (double)xa;
  acc[2] += dxheat_dzp;
  acc[3] += d4;
  acc[4] += (double)ts;
  acc[5] += (double)tk;
  acc[6] += (double)xn;
}

// ---------------------------------------------------------------------------
// shell z pass: for every shell r the c2r along z of its sfr and X-ray grids, accumulated per
// cell into the four evolveInt shell sums in registers over all shells, then stored once as a
// float4 per cell.  Two shells share one complex line (the two-for-one c2r of two real rows:
// shell r in the real part, shell r + 1 in the imaginary part; both rows are the same grid,
// filtered at neighbouring radii).
//
// Per shell: P_k[m], Q_k[m] (k = heat, ion, lya; m = x_e node) so that the cell's term is
// xray x (P_k[lo] + (x_e - X[lo]) Q_k[lo]), and cstar for max(sfr, 0); all scaled by a power of
// two per sum kind so FP32 keeps its range (the scale is undone in FP64 by the update kernel).

struct TsShellCoef {
  float P[3][x_int_NXHII];
  float Q[3][x_int_NXHII];
  float cstar;
  int kzmax;    // the shell's planes beyond this are zero (and not written)
  float dX[x_int_NXHII];   // widths of the node intervals
  // AGN units j = 0, 1 (the bands in use, soft first): max(grid, 0) x (PA + dx QA), with the
  // ratio of the band's prefactor to the galaxies' folded in so the terms join the same sums
  float PA[2][3][x_int_NXHII];
  float QA[2][3][x_int_NXHII];
};

struct TsZev {
  int nS;
  int m0, nm;                     // X-ray by nodes: the nodes m0 .. m0 + nm - 1 (nm 0: by shells)
  float X[x_int_NXHII];           // x_int_XHII (float, as in the reference)
  double inv_scale[4];            // undo the FP32 scaling
};

// LOOK: the pass's look-ups and sums per cell and shell: 0 none (X-ray by nodes, no AGN), 1 X-ray by shells, 2 AGN
// units. The default plan has one exchange at 16 values a thread at 128 and 256 (three blocks of 128
// threads, up to 168 registers); it is taken without look-ups, and by shells where a line takes 16 threads (256).
// Else 8 values a thread (two blocks of 256).  The passes over 40 shells, sharp-k unless it says top-hat, us at 8
// values a thread and in the one-exchange plan:
//   by nodes            128^3, 4 nodes 195 190; top-hat, 9 nodes 293 271     256^3, 2 nodes 1260 1140; top-hat, 9 2129 1831
//   by shells           128^3 303 315                                        256^3 2358 2360; top-hat 2917 2848
//   AGN, by nodes       128^3, 4 nodes 568 675                               256^3, 2 nodes 4277 4858; top-hat, 9 5692 6040
//   AGN, by shells      128^3 659 783                                        256^3 5330 6011
template <int N, int LOOK>
struct TsZ {
  static constexpr bool ONE = Plan<N>::S == 2 && N / Plan<N>::T == 16 && (LOOK == 0 || (LOOK == 1 && Plan<N>::T >= 16));
  using PL = std::conditional_t<ONE, Plan<N>, Plan8<N>>;
  static constexpr int T = PL::T;
  static constexpr int V = N / T;            // 8 or 16
  static constexpr int R0 = PL::R[0];
  static constexpr int Q = pow2_div(N, cmax((V == 16 ? 128 : 256) / T, 4));   // rows per block
  static constexpr int NTH = T * Q;
  static constexpr int MINB = V == 16 ? (NTH == 128 ? 3 : 1) : NTH >= 512 ? 1 : 512 / NTH;
  using Nodes = std::conditional_t<V == 16, uint64_t, uint32_t>;   // four bits a cell
  static constexpr int NZ = N / 2 + 1;
  // A shell's rows come as up to NBOX tensor boxes of KZS + 1 kz rows, KZS apart (they overlap in one
  // row, so every box lands on a 128-byte boundary and none leaves the spectrum): as many as the
  // shell's cut needs
  static constexpr int NBOX = N >= 64 ? 8 : 1;
  static constexpr int KZS = (N / 2) / NBOX;
  static constexpr int TS = round_up(NZ * Q, 16);            // one shell's rows, a 128-byte multiple
  static constexpr size_t tile_elems() { return (size_t)2 * TS; }   // two shells' rows
  static constexpr uint32_t BOX_TX = (uint32_t)((KZS + 1) * Q * sizeof(cf));
  static constexpr int STAGES = 3;           // tiles in flight: units u + 1 and u + 2 load during u
  static constexpr size_t smem() {
    return 128 + sizeof(cf) * (STAGES * tile_elems() + (size_t)line_buf_r0<N, R0, Q>() + N) +
           sizeof(uint64_t) * STAGES;
  }
  static_assert(Q % 2 == 0 && 2 * Q <= 256, "tensor box of 2Q floats, x a 16-byte multiple");
  static_assert(NBOX == 1 || (KZS * Q * sizeof(cf)) % 128 == 0, "boxes off a 128-byte boundary");
};

constexpr int TS_TMA_WAIT_LIMIT = 1 << 22;   // polls of an mbarrier before a wait gives up

// complex line of row q of the two spectra in a tile (a real part, b imaginary part), whose planes
// beyond ka and kb are zero; the tile holds tile[s][k][j] = (s ? b : a)[k][x][y0 + j], b at TS
template <int N, int Q, int TS>
__device__ __forceinline__ cf ts_tile_input(const cf* tile, int q, int p, int ka, int kb) {
  const int k = p <= N / 2 ? p : N - p;
  const cf A = k <= ka ? tile[k * Q + q] : cf{0.f, 0.f}, B = k <= kb ? tile[TS + k * Q + q] : cf{0.f, 0.f};
  if (p == 0 || p == N / 2) return cf{A.x, B.x};
  if (p < N / 2) return cf{A.x - B.y, A.y + B.x};
  return cf{A.x + B.y, B.x - A.y};
}

// Grids per shell: sfr, then with XS (X-ray by shells) the X-ray grid, then NA AGN bands (their
// per-cell heating terms also go to agn_heat, for the AGN heating averages).  Without XS the X-ray
// node fields follow the shells: heat, ion, lya of node zv.m0, then of the next node.
// The Hermitian column tiles arrive by tensor loads (the spectra as the tensor `tmap`: floats y
// innermost, then x, then kz of spectrum s at s (N/2 + 1) + kz), STAGES tiles in flight, one
// mbarrier each; a spectrum's planes beyond its cut are not loaded.
template <int N, bool XS, int NA>
__global__ void __launch_bounds__((TsZ<N, NA != 0 ? 2 : XS>::NTH), (TsZ<N, NA != 0 ? 2 : XS>::MINB))
    k_ts_zsum(const __grid_constant__ CUtensorMap tmap, const cf* __restrict__ g_tw,
              const TsShellCoef* __restrict__ gco, TsZev zv, const float* __restrict__ xe_prev,
              float4* __restrict__ sums, float2* __restrict__ agn_heat, uint32_t* err) {
  using Z = TsZ<N, NA != 0 ? 2 : XS>;
  using PL = typename Z::PL;
  constexpr int Q = Z::Q, V = Z::V, NZ = Z::NZ;
  constexpr int G = 1 + XS + NA;
  constexpr bool COEF = XS || NA > 0;   // units that read a pair's tables
  constexpr int PADW = 2 * (N / 2 + 1);
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  cf* tiles = reinterpret_cast<cf*>(sm);
  cf* xbuf = tiles + Z::STAGES * Z::tile_elems();
  cf* s_tw = xbuf + line_buf_r0<N, Z::R0, Q>();
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_tw + N);
  __shared__ TsShellCoef sc[COEF ? 2 : 1];
  const int x = blockIdx.y, y = blockIdx.x * Q + threadIdx.x % Q;
  const int t = threadIdx.x / Q;
  if (threadIdx.x == 0) {
    for (int b = 0; b < Z::STAGES; ++b) mbar_init(&bars[b], 1);
    mbar_init_fence();
  }
  load_twiddles_p<PL>(s_tw, g_tw);
  const size_t row = (size_t)x * N + y;
  // this thread's cells: z = last_pos(t, s); x_e interpolation node and offset
  // (ComputeTs.c:1198-1209): by shells the offset itself, by nodes its share of the interval
  float dxe[V];
  typename Z::Nodes lopack = 0;
  using Nodes = typename Z::Nodes;
#pragma unroll
  for (int sl = 0; sl < V; ++sl) {
    double xc = (double)__ldg(xe_prev + row * PADW + last_pos<PL>(t, sl));
    if (xc > (double)zv.X[x_int_NXHII - 1] * 0.999)
      xc = (double)zv.X[x_int_NXHII - 1] * 0.999;
    else if (xc < (double)zv.X[0])
      xc = 1.001 * (double)zv.X[0];
    // locate_xHII_index: the last node not above x_e (constant indices keep zv in the
    // parameter bank)
    const float xf = (float)xc;
    int m = 0;
    float xm = zv.X[0], xn = zv.X[1];
#pragma unroll
    for (int j = 1; j < x_int_NXHII; ++j)
      if (!(xf < zv.X[j])) {
        m = j;
        xm = zv.X[j];
        xn = zv.X[j + 1 < x_int_NXHII ? j + 1 : j];
      }
    lopack |= (Nodes)m << (4 * sl);
    dxe[sl] = XS ? (float)(xc - (double)xm) : (float)((xc - (double)xm) / ((double)xn - (double)xm));
  }
  // every thread's cells each on one x_e node of their own (the common case early in
  // reionization): the coefficient reads leave the per-cell loops.  The choice is the block's, as
  // both paths run transforms with block barriers.
  static_assert(V == 8 || V == 16, "the cells' x_e node indices in one word");
  const uint32_t lo0 = (uint32_t)lopack & 15u;
  bool uni = false;
  if constexpr (XS) uni = __syncthreads_and(lopack == (Nodes)(lo0 * 0x1111111111111111ull)) != 0;
  float a_heat[V], a_ion[V], a_lya[V], a_star[V];
  float a_agn0[NA > 0 ? V : 1], a_agn1[NA > 1 ? V : 1];
#pragma unroll
  for (int sl = 0; sl < V; ++sl) a_heat[sl] = a_ion[sl] = a_lya[sl] = a_star[sl] = 0.f;
#pragma unroll
  for (int sl = 0; sl < (NA > 0 ? V : 1); ++sl) a_agn0[sl] = 0.f;
#pragma unroll
  for (int sl = 0; sl < (NA > 1 ? V : 1); ++sl) a_agn1[sl] = 0.f;
  auto addr = [&](int p) { return line_addr_r0<Z::R0, Q>(p, threadIdx.x % Q); };
  // Units, two spectra each: u = G (r / 2) + g < nsh, the pair of shells (r, r + 1) of grid g; then
  // without XS one unit (heat, ion) per node, then one (lya, lya) per two nodes.  The tiles of units
  // u + 1 and u + 2 load while unit u is transformed (three buffers).  A missing second spectrum (an
  // odd count) reads as zeros.
  constexpr int S = Z::STAGES;
  const int y0 = blockIdx.x * Q, q = threadIdx.x % Q;
  const int nsh = G * ((zv.nS + 1) / 2), nm = XS ? 0 : zv.nm;
  const int nunits = nsh + nm + (nm + 1) / 2;
  // the spectra of unit u and the last plane of each (-1: there is none)
  auto unit = [&](int u, int (&sp)[2], int (&kl)[2]) {
    if (XS || u < nsh) {
      const int r = 2 * (u / G), g = u % G;
      const bool two = r + 1 < zv.nS;
      sp[0] = r * G + g;
      sp[1] = sp[0] + G;
      kl[0] = __ldg(&gco[r].kzmax);
      kl[1] = two ? __ldg(&gco[r + 1].kzmax) : -1;
    } else {
      const int v = u - nsh, base = zv.nS * G;
      const bool la = v >= nm;
      sp[0] = la ? base + 6 * (v - nm) + 2 : base + 3 * v;
      sp[1] = la ? sp[0] + 3 : sp[0] + 1;
      kl[0] = N / 2;
      kl[1] = !la || 2 * (v - nm) + 1 < nm ? N / 2 : -1;
    }
  };
  auto boxes = [](int k) { return k < 0 ? 0 : k <= Z::KZS ? 1 : (k + Z::KZS - 1) / Z::KZS; };
  // thread 0: tensor loads of unit u into its buffer
  auto issue = [&](int u) {
    const int b = u % S;
    int sp[2], kl[2];
    unit(u, sp, kl);
    mbar_arrive_expect_tx(&bars[b], (uint32_t)(boxes(kl[0]) + boxes(kl[1])) * Z::BOX_TX);
    for (int sh = 0; sh < 2; ++sh)
      for (int k = 0; k < boxes(kl[sh]); ++k)
        tma_load_3d(tiles + b * Z::tile_elems() + sh * Z::TS + k * Z::KZS * Q, &tmap, 2 * y0, x,
                    sp[sh] * NZ + k * Z::KZS, &bars[b]);
  };
  __syncthreads();   // barriers initialised
  if (threadIdx.x == 0)
    for (int u = 0; u < S - 1 && u < nunits; ++u) issue(u);
  bool waited = true;
  // the unit in work
  const cf* tile = tiles;
  int sp[2] = {0, 0}, kl[2] = {0, 0};
  auto input = [&](int p, int) { return ts_tile_input<N, Q, Z::TS>(tile, q, p, kl[0], kl[1]); };
  // an AGN unit j: clamped at 0 (ComputeTs.c:615-630), its own band tables
  auto agn_unit = [&](int j, float (&ah)[NA > 0 ? V : 1]) {
    line_fft_p<PL, true>(
        t, xbuf, s_tw, input, addr,
        [&](int, cf v, int sl) {
          const int lo = (int)((lopack >> (4 * sl)) & 15u);
          // by nodes dxe is the share of the interval, which the tables' slopes know as X
          const float d = XS ? dxe[sl] : dxe[sl] * sc[0].dX[lo];
          const float vx = fmaxf(v.x, 0.f), vy = fmaxf(v.y, 0.f);
          const float h = vx * fmaf(d, sc[0].QA[j][0][lo], sc[0].PA[j][0][lo]) +
                          vy * fmaf(d, sc[1].QA[j][0][lo], sc[1].PA[j][0][lo]);
          a_heat[sl] += h;
          ah[sl] += h;
          a_ion[sl] += vx * fmaf(d, sc[0].QA[j][1][lo], sc[0].PA[j][1][lo]) +
                       vy * fmaf(d, sc[1].QA[j][1][lo], sc[1].PA[j][1][lo]);
          a_lya[sl] += vx * fmaf(d, sc[0].QA[j][2][lo], sc[0].PA[j][2][lo]) +
                       vy * fmaf(d, sc[1].QA[j][2][lo], sc[1].PA[j][2][lo]);
        });
  };
  // the share of node m (counted from 0) in this thread's cell sl
  auto share = [&](int m, int sl) {
    const int lo = (int)((lopack >> (4 * sl)) & 15u);
    return lo == m ? 1.f - dxe[sl] : lo + 1 == m ? dxe[sl] : 0.f;
  };
  for (int u = 0; u < nunits; ++u) {
    const int r = 2 * (u / G), g = u % G;
    if (COEF && g == 0 && u < nsh) {
      __syncthreads();  // readers of the previous pair's coefficients are done
      const bool two = r + 1 < zv.nS;
      const int* src = reinterpret_cast<const int*>(gco + r);
      int* dst = reinterpret_cast<int*>(sc);
      // words per shell: the AGN tables only when there are AGN units
      constexpr int SW = (int)(sizeof(TsShellCoef) / sizeof(int));
      constexpr int W = NA > 0 ? SW : (int)(offsetof(TsShellCoef, PA) / sizeof(int));
      for (int i = threadIdx.x; i < 2 * W; i += Z::NTH) {
        const int sh = i / W, w = sh * SW + i % W;
        dst[w] = (sh == 0 || two) ? src[w] : 0;
      }
    }
    // buffer (u + 2) % 3 was consumed by unit u - 1 (the barrier at the end of its iteration)
    if (u + S - 1 < nunits && threadIdx.x == 0) issue(u + S - 1);
    if (!mbar_wait(&bars[u % S], (uint32_t)((u / S) & 1), TS_TMA_WAIT_LIMIT)) waited = false;
    if (COEF) __syncthreads();  // the pair's coefficients are visible to every thread
    tile = tiles + (u % S) * Z::tile_elems();
    unit(u, sp, kl);
    if (!XS && u >= nsh) {
      const int v = u - nsh;
      if (v < nm) {
        const int m = zv.m0 + v;
        line_fft_p<PL, true>(t, xbuf, s_tw, input, addr, [&](int, cf f, int sl) {
          const float w = share(m, sl);
          a_heat[sl] = fmaf(w, f.x, a_heat[sl]);
          a_ion[sl] = fmaf(w, f.y, a_ion[sl]);
        });
      } else {
        const int m = zv.m0 + 2 * (v - nm);
        line_fft_p<PL, true>(t, xbuf, s_tw, input, addr, [&](int, cf f, int sl) {
          a_lya[sl] += share(m, sl) * f.x + share(m + 1, sl) * f.y;
        });
      }
    } else if (g == 0) {
      // sfr: stellar Lyman-alpha sum, SFR clamped at 0 (ComputeTs.c:700)
      const float c0 = __ldg(&gco[r].cstar), c1 = kl[1] >= 0 ? __ldg(&gco[r + 1].cstar) : 0.f;
      line_fft_p<PL, true>(t, xbuf, s_tw, input, addr,
                           [&](int, cf v, int sl) { a_star[sl] += fmaxf(v.x, 0.f) * c0 + fmaxf(v.y, 0.f) * c1; });
    } else if (XS && g == 1) {
      // X-ray: heating, ionisation and Lyman-alpha integrands, not clamped
      if (uni) {
        // every cell of this thread on the same x_e node: its twelve coefficients read once
        float c[2][3][2];
#pragma unroll
        for (int sh = 0; sh < 2; ++sh)
#pragma unroll
          for (int kd = 0; kd < 3; ++kd) {
            c[sh][kd][0] = sc[sh].P[kd][lo0];
            c[sh][kd][1] = sc[sh].Q[kd][lo0];
          }
        line_fft_p<PL, true>(
            t, xbuf, s_tw, input, addr,
            [&](int, cf v, int sl) {
              const float d = dxe[sl];
              a_heat[sl] += v.x * fmaf(d, c[0][0][1], c[0][0][0]) + v.y * fmaf(d, c[1][0][1], c[1][0][0]);
              a_ion[sl] += v.x * fmaf(d, c[0][1][1], c[0][1][0]) + v.y * fmaf(d, c[1][1][1], c[1][1][0]);
              a_lya[sl] += v.x * fmaf(d, c[0][2][1], c[0][2][0]) + v.y * fmaf(d, c[1][2][1], c[1][2][0]);
            });
      } else {
        line_fft_p<PL, true>(
            t, xbuf, s_tw, input, addr,
            [&](int, cf v, int sl) {
              const int lo = (int)((lopack >> (4 * sl)) & 15u);
              const float d = dxe[sl];
              a_heat[sl] +=
                  v.x * fmaf(d, sc[0].Q[0][lo], sc[0].P[0][lo]) + v.y * fmaf(d, sc[1].Q[0][lo], sc[1].P[0][lo]);
              a_ion[sl] +=
                  v.x * fmaf(d, sc[0].Q[1][lo], sc[0].P[1][lo]) + v.y * fmaf(d, sc[1].Q[1][lo], sc[1].P[1][lo]);
              a_lya[sl] +=
                  v.x * fmaf(d, sc[0].Q[2][lo], sc[0].P[2][lo]) + v.y * fmaf(d, sc[1].Q[2][lo], sc[1].P[2][lo]);
            });
      }
    } else if constexpr (NA > 0) {
      if (g == 1 + XS) {
        agn_unit(0, a_agn0);
      } else if constexpr (NA > 1) {
        agn_unit(1, a_agn1);
      }
    }
    // the tile is consumed (generic reads ordered before the tensor load that refills it)
    fence_proxy_async_smem();
    __syncthreads();
  }
  if (!waited && threadIdx.x % 32 == 0) atomicExch(err, 1u);
#pragma unroll
  for (int sl = 0; sl < V; ++sl) {
    const size_t ic = row * N + last_pos<PL>(t, sl);
    sums[ic] = make_float4(a_heat[sl], a_ion[sl], a_lya[sl], a_star[sl]);
    if constexpr (NA > 0) agn_heat[ic] = make_float2(a_agn0[sl], NA > 1 ? a_agn1[NA > 1 ? sl : 0] : 0.f);
  }
}

// the per-cell update (ComputeTs.c:1171-1407) from the shell sums; sums == nullptr: no light.  Cells
// in memory order whatever the row length (a block per row left half of its threads idle at 128^3);
// bound by its FP64 work, three exponentials, two logarithms, a cube root and the iteration a cell.
// With the iteration on 1 / T_S, the scalars as parameters and the tables' index: 8.35 -> 7.25 ms at
// 512^3, 0.25 -> 0.125 at 128^3.
constexpr int EV_NT = 128;
__global__ void __launch_bounds__(EV_NT, 5) k_ts_evolve(const TsDev* __restrict__ gC, const TsPar P, const TsEvolve e,
                                                        double4 inv_scale, int n, const float4* __restrict__ sums,
                                                        const float2* __restrict__ agn_heat,
                                                        const float* __restrict__ deltax, float* __restrict__ xe_prev,
                                                        float* __restrict__ xe_box, float* __restrict__ Tk,
                                                        float* __restrict__ TS, double* __restrict__ partials,
                                                        int* __restrict__ nonconv, const uint32_t* __restrict__ err) {
  if (err && *err) return;   // a tile's wait ran out: the sums are not to be used, the state stays
  __shared__ TsDev C;
  {
    const int* src = reinterpret_cast<const int*>(gC);
    int* dst = reinterpret_cast<int*>(&C);
    for (int i = threadIdx.x; i < (int)(sizeof(TsDev) / sizeof(int)); i += EV_NT) dst[i] = src[i];
  }
  __syncthreads();
  const size_t n3 = (size_t)n * n * n;
  double acc[TS_NSUM];
#pragma unroll
  for (int i = 0; i < TS_NSUM; ++i) acc[i] = 0.0;
  int nc = 0;
  for (size_t ir = (size_t)blockIdx.x * EV_NT + threadIdx.x; ir < n3; ir += (size_t)gridDim.x * EV_NT) {
    const size_t ip = ir + ((unsigned)ir / (unsigned)n) * 2;   // rows of n + 2 values
    double sm[4] = {0.0, 0.0, 0.0, 0.0};
    if (sums) {
      const float4 v = __ldg(sums + ir);
      sm[0] = (double)v.x * inv_scale.x;
      sm[1] = (double)v.y * inv_scale.y;
      sm[2] = (double)v.z * inv_scale.z;
      sm[3] = (double)v.w * inv_scale.w;
    }
    float xn, tk, ts;
    const float xe0 = xe_prev[ip];
    if (agn_heat) {
      // the AGN heating terms of dT_K/dz (XRayHeatingFunctions.c:1519-1520) for their averages
      const float2 a = __ldg(agn_heat + ir);
      const double f = inv_scale.x * e.const_zp * e.heat_conv / (1.0 + (double)xe0);
      acc[7] += (double)a.x * f;
      acc[8] += (double)a.y * f;
    }
    evolve_cell(C, P, e, __ldg(deltax + ip), xe0, Tk[ir], sm, &xn, &tk, &ts, acc, &nc);
    xe_prev[ip] = xn;
    xe_box[ip] = xn;
    Tk[ir] = tk;
    TS[ir] = ts;
  }
  if (nc) atomicAdd(nonconv, nc);
  block_sum_dyn<TS_NSUM>(acc, partials + (size_t)blockIdx.x * TS_NSUM);
}

// homogeneous branch (ComputeTs.c:252-278) and the closing averages (:1459-1494)
__global__ void __launch_bounds__(256) k_ts_homog(const TsDev* __restrict__ gC, const TsPar P, float xe0, float TK0,
                                                  float cT_ad, int n, const float* __restrict__ deltax,
                                                  float* __restrict__ xe_prev, float* __restrict__ xe_box,
                                                  float* __restrict__ Tk, float* __restrict__ TS,
                                                  double* __restrict__ partials, int* __restrict__ nonconv) {
  __shared__ TsDev C;
  {
    const int* src = reinterpret_cast<const int*>(gC);
    int* dst = reinterpret_cast<int*>(&C);
    for (int i = threadIdx.x; i < (int)(sizeof(TsDev) / sizeof(int)); i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  const int padw = 2 * (n / 2 + 1);
  const size_t rows = (size_t)n * n;
  double acc[TS_NSUM];
#pragma unroll
  for (int i = 0; i < TS_NSUM; ++i) acc[i] = 0.0;
  int nc = 0;
  for (size_t row = blockIdx.x; row < rows; row += gridDim.x)
    for (int z = threadIdx.x; z < n; z += blockDim.x) {
      const size_t ir = row * n + z, ip = row * padw + z;
      const float delta = deltax[ip];
      const float tk = (float)((double)TK0 * (1.0 + (double)(cT_ad * delta)));
      float xa;
      const float ts = get_Ts(C, P, delta, tk, xe0, 0.f, &xa, &nc);
      xe_prev[ip] = xe0;
      xe_box[ip] = xe0;
      Tk[ir] = tk;
      TS[ir] = ts;
      acc[4] += (double)ts;
      acc[5] += (double)tk;
      acc[6] += (double)xe0;
    }
  if (nc) atomicAdd(nonconv, nc);
  block_sum_dyn<TS_NSUM>(acc, partials + (size_t)blockIdx.x * TS_NSUM);
}

// ---------------------------------------------------------------------------
// host side

// knots (log T, log kappa) and per-interval coefficients of one kappa table
static void fill_spline(const CubicSpline& sp, const std::vector<double>& lx, const std::vector<double>& ly,
                        KappaSpline* k) {
  std::memset(k, 0, sizeof(*k));
  k->n = (int)lx.size();
  for (int i = 0; i < k->n; ++i) {
    k->x[i] = lx[i];
    k->y[i] = ly[i];
    if (i + 1 < k->n) {
      double a;
      sp.coeffs((size_t)i, &a, &k->b[i], &k->c[i], &k->d[i]);
    }
  }
  const double step = (lx.back() - lx[0]) / KLUT;
  k->x0 = lx[0];
  k->inv_step = 1.0 / step;
  for (int s = 0, lo = 0; s < KLUT; ++s) {
    // (a knot within rounding of the step's start is left to the device's search)
    while (lo < k->n - 2 && lx[lo + 1] < lx[0] + (s - 1e-6) * step) ++lo;
    k->lut[s] = lo;
  }
}

// The combination of a shell that reads more than TS_MAXSRC history slots:
// spec[spare][g] = sum_i cs[i] spec[ks[i]][g] for every grid g, accumulated with fmaf in the order
// of i as the x pass does (1 x value is exact, so the shell's x pass then reads the same numbers).
// Sources go in chunks of TS_COMB; later chunks continue from the partial sums.
constexpr int TS_COMB = 32;
struct TsComb {
  int n;
  int first;   // the chunk starts the sums (else it adds to the spare slot)
  int ks[TS_COMB];
  float cs[TS_COMB];
};

__global__ void __launch_bounds__(256) k_ts_combine(cf* __restrict__ spec, size_t stride, int G, TsComb cb,
                                                    int spare) {
  const size_t total = stride * (size_t)G;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    const size_t g = e / stride, i = e - g * stride;
    cf* out = spec + ((size_t)spare * G + g) * stride + i;
    float ax = 0.f, ay = 0.f;
    if (!cb.first) {
      ax = out->x;
      ay = out->y;
    }
    for (int k = 0; k < cb.n; ++k) {
      const cf v = spec[((size_t)cb.ks[k] * G + g) * stride + i];
      ax = fmaf(cb.cs[k], v.x, ax);
      ay = fmaf(cb.cs[k], v.y, ay);
    }
    *out = cf{ax, ay};
  }
}

static int ts_combine(rg_context* ctx, int n, cf* spec, size_t stride, int G, const std::vector<int>& ks,
                      const std::vector<float>& cs, int spare, cudaStream_t st) {
  (void)n;
  const int blocks = 4 * ctx->num_sms;
  for (size_t i0 = 0; i0 < ks.size(); i0 += TS_COMB) {
    TsComb cb;
    std::memset(&cb, 0, sizeof(cb));
    cb.first = i0 == 0;
    cb.n = (int)std::min((size_t)TS_COMB, ks.size() - i0);
    for (int k = 0; k < cb.n; ++k) {
      cb.ks[k] = ks[i0 + k];
      cb.cs[k] = cs[i0 + k];
    }
    prof_begin(ctx, "ts_combine_sources", st);
    k_ts_combine<<<blocks, 256, 0, st>>>(spec, stride, G, cb, spare);
    prof_end(ctx, 8.0 * stride * G * (cb.n + (cb.first ? 1 : 2)), st);
    RG_CUDA_TRY(ctx, cudaGetLastError());
  }
  return RG_OK;
}

// x and y passes of a batch of shells: work_base + (j * bt.ng + g) * stride, j < bt.nr.  (The
// fused x/y kernel of find_HII_bubbles, run on these batches, measured slower at 512^3: 48.8 ms
// against 43.5 ms for the two passes; the x pass here reads its history spectra mostly from L2.)
template <int N>
static int launch_ts_xy(rg_context* ctx, const cf* spec, cf* work_base, size_t stride, TsBatch& bt,
                        const float* wtab, int wpitch, cudaStream_t st) {
  using C = Cfg<N>;
  const cf* tw;
  int rc = twiddles_for(ctx, N, &tw);
  if (rc) return rc;
  // planes the batch has, and the modes and columns its shells keep (for the algorithmic bytes)
  int kzmax = 0;
  double src_reads = 0, cols = 0, lines = 0;
  const double full = (double)C::NZ * N * N;
  for (int r = 0; r < bt.nr; ++r) {
    const double k = std::sqrt((double)bt.cut[r]);
    const int kz = std::min(N / 2, (int)k);
    kzmax = std::max(kzmax, kz);
    src_reads += bt.nk[r] * std::min(full, 2.0 / 3.0 * M_PI * k * k * k);
    cols += std::min(full, M_PI / 2 * k * k * N);
    lines += std::min(full, (kz + 1.0) * N * N);
  }
  const size_t smx = sizeof(cf) * (N + (size_t)line_buf<N, C::BX>());
  RG_CUDA_TRY(ctx, cudaFuncSetAttribute(k_ts_x<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smx));
  prof_begin(ctx, "ts_x_c2c_combine_window", st);
  // A block takes up to 8 shells, which mostly combine the same sources; fewer where that leaves under 8
  // blocks an SM.  40 shells of 3 grids at 64^3, x and y passes with the frequency integrals running
  // beside: 216 us in one launch each of 2 shells a block, 321 in five launches of 8.
  const int per_shell = (N / C::BX) * (kzmax + 1);
  bt.chunk = std::min(TS_KB, std::max(1, bt.nr * per_shell / (8 * ctx->num_sms)));
  k_ts_x<N><<<dim3(N / C::BX, kzmax + 1, (bt.nr + bt.chunk - 1) / bt.chunk), C::T * C::BX, smx, st>>>(spec, stride, work_base, bt, wtab, wpitch, tw);
  prof_end(ctx, bt.ng * 8.0 * (src_reads + cols), st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  using Y = YCfg<N>;
  RG_CUDA_TRY(ctx, cudaFuncSetAttribute(k_ts_y<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Y::smem()));
  prof_begin(ctx, "ts_y_c2c", st);
  k_ts_y<N><<<dim3(N / Y::BY, kzmax + 1, bt.ng * bt.nr), Y::NTH, Y::smem(), st>>>(work_base, stride, bt, tw);
  prof_end(ctx, bt.ng * 8.0 * (cols + lines), st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  return RG_OK;
}

// the X-ray node fields: their spectra, then the inverse x and y passes in place
template <int N>
static int launch_ts_nodes(rg_context* ctx, const cf* spec, cf* fields, size_t stride, int gs,
                           const TsNodeShell* d_sh, int nS, int nm, const float* wtab, int wpitch, cudaStream_t st) {
  using C = Cfg<N>;
  const cf* tw;
  int rc = twiddles_for(ctx, N, &tw);
  if (rc) return rc;
  const int nf = 3 * nm, log2n = __builtin_ctz(N);
  const int per = ts_node_chunk(nm);
  const dim3 grid((unsigned)std::min((stride + 255) / 256, (size_t)ctx->num_sms * 64), ts_node_chunks(nm));
  prof_begin(ctx, "ts_xray_nodes", st);
  if (per == 2)
    k_ts_nodes<6><<<grid, 256, 0, st>>>(spec, stride, gs, fields, d_sh, nS, nf, wtab, wpitch, log2n);
  else if (per == 3)
    k_ts_nodes<9><<<grid, 256, 0, st>>>(spec, stride, gs, fields, d_sh, nS, nf, wtab, wpitch, log2n);
  else
    k_ts_nodes<12><<<grid, 256, 0, st>>>(spec, stride, gs, fields, d_sh, nS, nf, wtab, wpitch, log2n);
  prof_end(ctx, 8.0 * stride * nf, st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  const size_t smx = sizeof(cf) * (N + (size_t)line_buf<N, C::BX>());
  RG_CUDA_TRY(ctx, cudaFuncSetAttribute(k_pass_x<N, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smx));
  prof_begin(ctx, "ts_nodes_x_c2c", st);
  k_pass_x<N, true><<<dim3(N / C::BX, C::NZ, nf), C::T * C::BX, smx, st>>>(fields, stride, tw, 1.f);
  prof_end(ctx, 16.0 * stride * nf, st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  prof_begin(ctx, "ts_nodes_y_c2c", st);
  RG_CUDA_TRY(ctx, (launch_pass_y<N, true>(fields, stride, nf, tw, st)));
  prof_end(ctx, 16.0 * stride * nf, st);
  return RG_OK;
}

// the z pass over all nS shells (and the node fields): per-cell shell sums
template <int N, bool XS, int NA>
static int launch_ts_zsum_g(rg_context* ctx, const cf* work, size_t stride, const TsShellCoef* d_co, const TsZev& zv,
                            const float* xe_prev, float4* sums, float2* agn_heat, double planes, cudaStream_t st) {
  const cf* tw;
  int rc = twiddles_for(ctx, N, &tw);
  if (rc) return rc;
  using Z = TsZ<N, NA != 0 ? 2 : XS>;
  const double n3 = (double)N * N * N;
  if (stride != (size_t)Z::NZ * N * N) return set_error(ctx, RG_EINVAL, "Ts z pass: shell spectra must be contiguous");
  // every spectrum (S[kz][x][y], one after another) as a 3-D float tensor
  CUtensorMap tmap;
  const uint64_t dims[3] = {2ull * N, (uint64_t)N, (uint64_t)Z::NZ * (zv.nS * (1 + XS + NA) + (XS ? 0 : 3 * zv.nm))};
  const uint64_t strides[2] = {8ull * N, 8ull * N * N};
  const uint32_t box[3] = {2u * Z::Q, 1u, (uint32_t)Z::KZS + 1u};
  const int mrc = tma_map_3d(&tmap, work, dims, strides, box);
  if (mrc != 0) return set_error(ctx, RG_ECUDA, "cuTensorMapEncodeTiled failed (" + std::to_string(mrc) + ")");
  const size_t smz = Z::smem();
  RG_CUDA_TRY(ctx, cudaFuncSetAttribute(k_ts_zsum<N, XS, NA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smz));
  prof_begin(ctx, "ts_z_c2r_sums", st);
  k_ts_zsum<N, XS, NA><<<dim3(N / Z::Q, N), Z::NTH, smz, st>>>(tmap, tw, d_co, zv, xe_prev, sums, agn_heat,
                                                                ctx->xy_ctrl);
  // the planes of the spectra, x_e read, four float sums (and the AGN heating pair) written
  prof_end(ctx, planes * 8.0 * N * N + 4.0 * n3 + 16.0 * n3 + (NA > 0 ? 8.0 * n3 : 0.0), st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  return RG_OK;
}

template <int N>
static int launch_ts_zsum(rg_context* ctx, const cf* work, size_t stride, int nagn, const TsShellCoef* d_co,
                          const TsZev& zv, const float* xe_prev, float4* sums, float2* agn_heat, double planes,
                          cudaStream_t st) {
#define RG_TS_Z(XS, NA) launch_ts_zsum_g<N, XS, NA>(ctx, work, stride, d_co, zv, xe_prev, sums, agn_heat, planes, st)
  if (zv.nm) return nagn == 0 ? RG_TS_Z(false, 0) : nagn == 1 ? RG_TS_Z(false, 1) : RG_TS_Z(false, 2);
  return nagn == 0 ? RG_TS_Z(true, 0) : nagn == 1 ? RG_TS_Z(true, 1) : RG_TS_Z(true, 2);
#undef RG_TS_Z
}

#define RG_TS_DISPATCH(n, call)                                                           \
  switch (n) {                                                                            \
    case 8: { constexpr int NN = 8; return call; }                                        \
    case 16: { constexpr int NN = 16; return call; }                                      \
    case 32: { constexpr int NN = 32; return call; }                                      \
    case 64: { constexpr int NN = 64; return call; }                                      \
    case 128: { constexpr int NN = 128; return call; }                                    \
    case 256: { constexpr int NN = 256; return call; }                                    \
    case 512: { constexpr int NN = 512; return call; }                                    \
    default: return set_error(ctx, RG_EUNSUPPORTED, "ComputeTs needs a power-of-two ReionGridDim"); \
  }

static int ts_xy(rg_context* ctx, int n, const cf* spec, cf* work_base, size_t stride, TsBatch& bt,
                 const float* wtab, int wpitch, cudaStream_t st) {
  RG_TS_DISPATCH(n, launch_ts_xy<NN>(ctx, spec, work_base, stride, bt, wtab, wpitch, st));
}

static int ts_nodes(rg_context* ctx, int n, const cf* spec, cf* fields, size_t stride, int gs, const TsNodeShell* d_sh,
                    int nS, int nm, const float* wtab, int wpitch, cudaStream_t st) {
  RG_TS_DISPATCH(n, launch_ts_nodes<NN>(ctx, spec, fields, stride, gs, d_sh, nS, nm, wtab, wpitch, st));
}

static int ts_zsum(rg_context* ctx, int n, const cf* work, size_t stride, int nagn, const TsShellCoef* d_co,
                   const TsZev& zv, const float* xe_prev, float4* sums, float2* agn_heat, double planes,
                   cudaStream_t st) {
  RG_TS_DISPATCH(n, launch_ts_zsum<NN>(ctx, work, stride, nagn, d_co, zv, xe_prev, sums, agn_heat, planes, st));
}

// the last n2 that the sharp-k window of radius R keeps (k R 0.413566994 > 1 drops a mode)
static int sharpk_cut(double delta_k, double R, int n2max) {
  auto drops = [&](int n2) { return delta_k * std::sqrt((double)n2) * R * 0.413566994 > 1.0; };
  int lo = 0, hi = n2max + 1;   // lo is kept; hi is dropped, or past the table
  while (hi > lo + 1) {
    const int mid = (lo + hi) / 2;
    if (drops(mid))
      hi = mid;
    else
      lo = mid;
  }
  return lo;
}

// the cuts of the shells' windows: sharp-k, without the first shell, which is not filtered (ComputeTs.c:529)
static std::vector<int> ts_cuts(const rg_params* p, const TsShells& sh, int n2max) {
  std::vector<int> cut(sh.nS, TS_NOCUT);
  if (p->TsHeatingFilterType == 1)
    for (int r = 1; r < sh.nS; ++r) cut[r] = sharpk_cut(2.0 * M_PI / p->BoxSize, sh.R[r], n2max);
  return cut;
}

// a shell combines more than TS_MAXSRC history snapshots
static bool ts_wide(const TsShells& sh) {
  for (int r = 0; r < sh.nS; ++r) {
    int nk = 0;
    for (int k = 0; k < sh.nsrc; ++k) nk += sh.coef[(size_t)r * sh.nsrc + k] != 0.f;
    if (nk > TS_MAXSRC) return true;
  }
  return false;
}

// X-ray by nodes (m0 .. m0 + nm - 1, around the box's x_e, xe_lo to xe_hi, clamped as each cell's is) or
// by shells (nm 0), whichever costs less.  In units of a z unit (two spectra): a node takes three fields
// through k_ts_nodes and the x and y passes and 1.5 z units, 5.8 to 6.4 units measured at 128^3 to 512^3;
// a pair of shells a z unit with the table look-ups, 1.15 to 1.5, and a pass over what its window
// leaves, 0.42 a full one.  With 40 sharp-k shells the line lies between 4 and 6 nodes: 512^3 with 5
// nodes 24.8 ms by nodes and 21.8 by shells, 256^3 with 9 4.2 and 2.9, 128^3 with 4 0.53 and 0.61.
// A shell with its combination in a spare slot, which later batches overwrite, and a NaN in x_e
// keep the shells.
static void ts_choose_nodes(const float* X, int N, const std::vector<int>& cut, bool wide, float xe_lo, float xe_hi,
                            int* m0, int* nm) {
  *m0 = *nm = 0;
  if (wide || std::isnan(xe_lo) || std::isnan(xe_hi)) return;
  auto node = [&](float v) {
    const double top = (double)X[x_int_NXHII - 1] * 0.999;
    const double xc = (double)v > top ? top : (double)v < (double)X[0] ? 1.001 * (double)X[0] : (double)v;
    return locate_xHII_index(X, (float)xc);
  };
  const int first = node(xe_lo), count = node(xe_hi) + 2 - first;
  double passes = 0;
  for (int c : cut) {
    const double k = std::sqrt((double)c) / (N / 2);
    passes += std::min(1.0, M_PI / 4 * k * k) + std::min(1.0, k);
  }
  if (6.0 * count >= 1.25 * (0.5 * cut.size()) + 0.42 * passes) return;
  *m0 = first;
  *nm = count;
}

void ts_debug_nodes(const rg_params* p, const TsShells& sh, const float* X, float xe_lo, float xe_hi, int* out) {
  const int N = p->ReionGridDim;
  ts_choose_nodes(X, N, ts_cuts(p, sh, 3 * (N / 2) * (N / 2)), ts_wide(sh), xe_lo, xe_hi, &out[0], &out[1]);
  out[2] = out[1] ? ts_node_chunks(out[1]) : 0;
  out[3] = out[1] ? ts_node_reads(out[1]) : 0;
  out[4] = (int)(sizeof(TsNodeShell::f) / sizeof(float));
}

static double pow2_scale(double maxabs) {
  if (!(maxabs > 0) || !std::isfinite(maxabs)) return 1.0;
  return std::ldexp(1.0, -std::ilogb(maxabs));
}

int ts_snapshot(rg_context* ctx, const rg_params* p, const rg_snapshot* s, const rg_grids* g, rg_ts_scalars* out,
                const rg_grids* src_host, const Staging* stg) {
  int rc;
  const Staging none;
  if (!stg) stg = &none;
  bool kicked = false;
  auto kick = [&]() -> int {
    if (kicked || !stg->after_sources) return RG_OK;
    kicked = true;
    return stg->after_sources();
  };
  cudaStream_t st = ctx->stream;
  const int N = ctx->N;
  const size_t n3 = (size_t)N * N * N;
  const Cosmo cm(p);
  const Units u = make_units(p);
  const double zp = s->ZZ[s->snapshot];
  const double box_size = p->BoxSize / p->Hubble_h;  // Mpc
  const double pixel_volume = std::pow(box_size / (double)N, 3);
  std::memset(out, 0, sizeof(*out));
  // grids per shell: sfr, X-ray, then the AGN bands in use (0 soft, 1 hard)
  const int agn_flag = p->Flag_IncludeAGNXray;
  int bands[2] = {-1, -1}, nagn = 0;
  if (agn_flag == 1 || agn_flag == 3) bands[nagn++] = 0;
  if (agn_flag == 1 || agn_flag == 2) bands[nagn++] = 1;
  const int G = 2 + nagn;

  // device constants: kappa splines and number densities
  TsDev hc;
  std::memset(&hc, 0, sizeof(hc));
  fill_spline(ctx->tables.k10, ctx->tables.k10_lT, ctx->tables.k10_lk, &hc.k10);
  fill_spline(ctx->tables.kel, ctx->tables.kel_lT, ctx->tables.kel_lk, &hc.kel);
  fill_spline(ctx->tables.kpH, ctx->tables.kpH_lT, ctx->tables.kpH_lk, &hc.kpH);
  TsPar par;
  par.max_iter = ctx->ts_iter_limit;
  {
    // per-redshift factors of xcoll / taugp / xalpha_tilde / dT_comp / evolveInt; the C passes
    // the redshift to them as a float
    const float zf = (float)zp;
    const double z = (double)zf;
    TsZConst& Z = par.z;
    Z.Trad = TCMB * (1.0 + z);
    Z.inv_Trad = 1.0 / Z.Trad;
    const double opz3 = std::pow(1.0 + z, 3.0);
    Z.xc_H = T21 / Z.Trad * cm.No * opz3 / A10_HYPERFINE;
    Z.xc_e = T21 / Z.Trad * cm.N_b0 * opz3 / A10_HYPERFINE;
    Z.xc_p = Z.xc_H;
    Z.tgp0 = 1.342881e-7 / cm.hubble(zf) * cm.No * opz3;
    Z.xa0 = 1.66e11 / (1.0 + z);
    Z.nb0 = cm.N_b0 * std::pow((double)(1.0f + zf), 3);
    Z.comp0 = (-1.51e-4) / (cm.hubble(zf) / (HUBBLE * p->Hubble_h)) / p->Hubble_h * std::pow(Z.Trad, 4.0) / (1.0 + z);
    Z.dadia0 = 3 / (1.0 + z);
    Z.f_H = cm.f_H;
    Z.f_He = cm.f_He;
  }
  // device constants and the per-shell coefficients live in one context buffer:
  // [TsDev][TsShellCoef x shells][TsNodeShell x shells]
  const int nS_all = p->TsNumFilterSteps;
  const size_t off_co = (sizeof(TsDev) + 255) / 256 * 256;
  if ((rc = ensure_device(ctx, &ctx->ts_const, &ctx->ts_const_elems,
                          off_co + (sizeof(TsShellCoef) + sizeof(TsNodeShell)) * (nS_all + 1))))
    return rc;
  TsDev* d_hc = reinterpret_cast<TsDev*>(ctx->ts_const);
  TsStatus* d_status = reinterpret_cast<TsStatus*>(ctx->d_sums + TS_STATUS);
  TsShellCoef* d_co = reinterpret_cast<TsShellCoef*>(ctx->ts_const + off_co);
  RG_CUDA_TRY(ctx, cudaMemcpyAsync(d_hc, &hc, sizeof(TsDev), cudaMemcpyHostToDevice, st));
  TsNodeShell* d_node = reinterpret_cast<TsNodeShell*>(d_co + nS_all + 1);
  RG_CUDA_TRY(ctx, cudaMemsetAsync(d_status, 0, sizeof(TsStatus), st));
  // the sums and the status behind them, in one copy
  TsStatus status;
  auto fetch = [&]() -> int {
    RG_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_sums, ctx->d_sums, sizeof(double) * TS_STATUS + sizeof(TsStatus),
                                     cudaMemcpyDeviceToHost, st));
    return RG_OK;
  };
  const int nblk = 148 * 8;
  double* partials = ensure_partials(ctx, (size_t)nblk * TS_NSUM);
  if (!partials) return set_error(ctx, RG_ENOMEM, "partials");

  const double R0 = L_FACTOR * box_size / (float)N;
  const double Mh2 = rtom(p, R0) * p->Hubble_h * p->Hubble_h;
  const double ftpr3 = (4.0 / 3.0) * M_PI * std::pow(R0, 3.0) / pixel_volume;

  bool waits = false;   // kernels with device waits were launched
  auto finish = [&](bool homog, int nblocks) -> int {
    if ((rc = kick())) return rc;
    if ((rc = reduce_partials(ctx, partials, nblocks, TS_NSUM, ctx->d_sums, st))) return rc;
    if ((rc = fetch())) return rc;
    if (waits && (rc = xy_ctrl_fetch(ctx, st))) return rc;
    RG_CUDA_TRY(ctx, cudaStreamSynchronize(st));
    prof_resolve(ctx);
    if (waits && (rc = xy_ctrl_result(ctx))) return rc;
    std::memcpy(&status, ctx->h_sums + TS_STATUS, sizeof(status));
    const double* S = ctx->h_sums;
    const double nn = (double)n3;
    if (!homog) {
      out->volume_ave_J_alpha = S[0] / nn;
      out->volume_ave_xalpha = S[1] / nn;
      out->volume_ave_Xheat = S[2] / nn;
      out->volume_ave_Xion = S[3] / nn;
      for (int j = 0; j < nagn; ++j)
        (bands[j] ? out->volume_ave_Xheat_AGN_hard : out->volume_ave_Xheat_AGN_soft) = S[7 + j] / nn;
    }
    out->volume_ave_TS = S[4] / nn;
    out->volume_ave_TK = S[5] / nn;
    out->volume_ave_xe = S[6] / nn;
    out->homogeneous = homog;
    if (status.nonconv)
      return set_error(ctx, RG_ETIMEDOUT, "get_Ts did not converge in " + std::to_string(ctx->ts_iter_limit) +
                                              " iterations for some cells");
    return RG_OK;
  };

  // collapse fraction and <x_e> (both branches compute the collapse fraction)
  prof_begin(ctx, "ts_reduce0", st);
  if ((rc = stage_wait(ctx, stg->inputs, st))) return rc;
  k_ts_reduce0<<<nblk, 256, 0, st>>>(g->stars, g->deltax, g->x_e_box_prev, N, Mh2, ftpr3, partials, d_status);
  prof_end(ctx, 12.0 * n3, st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  if ((rc = reduce_partials(ctx, partials, nblk, 2, ctx->d_sums, st))) return rc;
  if ((rc = fetch())) return rc;
  RG_CUDA_TRY(ctx, cudaStreamSynchronize(st));
  const double collapse_fraction = ctx->h_sums[0] / (double)n3;
  const double x_e_ave = ctx->h_sums[1] / (double)n3;
  std::memcpy(&status, ctx->h_sums + TS_STATUS, sizeof(status));
  const float xe_lo = float_of_order(~status.xe_bottom), xe_hi = float_of_order(status.xe_top);
  out->collapse_fraction = collapse_fraction;
  out->x_e_ave = x_e_ave;

  if ((zp - p->ReionMaxHeatingRedshift) >= -0.0001) {
    const float xe0 = (float)xion_RECFAST(ctx->tables, (float)zp);
    const float TK0 = (float)T_RECFAST(ctx->tables, (float)zp);
    prof_begin(ctx, "ts_homog", st);
    if ((rc = stage_wait(ctx, stg->closing, st))) return rc;   // Tk_box is overwritten
    k_ts_homog<<<nblk, 256, 0, st>>>(d_hc, par, xe0, TK0, cT_approx((float)zp), N, g->deltax, g->x_e_box_prev,
                                      g->x_e_box, g->Tk_box, g->TS_box, partials, &d_status->nonconv);
    prof_end(ctx, 28.0 * n3, st);
    RG_CUDA_TRY(ctx, cudaGetLastError());
    return finish(true, nblk);
  }

  // inhomogeneous branch
  TsShells sh = ts_shells(p, s->ZZ, s->n_snapshots, s->snapshot, src_host ? src_host->n_hist : g->n_hist);
  if (sh.error) return set_error(ctx, RG_EINVAL, sh.msg);
  const int nS = sh.nS;
  const bool no_light = !(collapse_fraction > 0.0);
  const TsPrefactors pf = ts_prefactors(p, zp);
  const double prev_redshift = s->snapshot == 0 ? s->ZZ[s->snapshot] : s->ZZ[s->snapshot - 1];
  const size_t nc = (size_t)(N / 2 + 1) * N * N;
  const size_t npad = (size_t)N * N * 2 * (N / 2 + 1);
  TsZev zv;
  std::memset(&zv, 0, sizeof(zv));
  for (int m = 0; m < x_int_NXHII; ++m) zv.X[m] = ctx->tables.x_int_XHII[m];
  for (int k = 0; k < 4; ++k) zv.inv_scale[k] = 1.0;

  if (!no_light) {
    if (!s->stored_fcoll && s->snapshot > 0)
      return set_error(ctx, RG_EINVAL, "ComputeTs needs stored_fcoll of the previous snapshot");
    if ((rc = ts_freq_start(ctx, p, sh, zp, x_e_ave, collapse_fraction, s->ZZ, s->stored_fcoll, s->snapshot)))
      return rc;
    // sources used by any shell
    std::vector<int> slot_of(sh.nsrc, -1), used;
    for (int r = 0; r < nS; ++r)
      for (int k = 0; k < sh.nsrc; ++k)
        if (sh.coef[(size_t)r * sh.nsrc + k] != 0.f && slot_of[k] < 0) {
          slot_of[k] = (int)used.size();
          used.push_back(k);
        }
    // a shell that combines more than TS_MAXSRC history snapshots gets its combination formed
    // beforehand (k_ts_combine) into one of TS_KB spare slots after the used sources
    const bool wide = ts_wide(sh);
    const int nused = std::max(1, (int)used.size());
    // window cuts (filter() takes BoxSize in Mpc/h and R in Mpc, ComputeTs.c:532)
    const int n2max = 3 * (N / 2) * (N / 2);
    const bool sharp = p->TsHeatingFilterType == 1;
    const std::vector<int> cut = ts_cuts(p, sh, n2max);
    ts_choose_nodes(ctx->tables.x_int_XHII.data(), N, cut, wide, xe_lo, xe_hi, &zv.m0, &zv.nm);
    const int xs = zv.nm == 0;              // X-ray grids per shell
    const int Gs = 1 + xs + nagn;           // grids per shell
    const size_t slots = (size_t)nused + (wide ? TS_KB : 0);
    if ((rc = ensure_device(ctx, &ctx->spec, &ctx->spec_elems, nc * G * slots))) return rc;
    // every shell's filtered grids stay in HBM until the fused z pass (G nS spectra)
    if ((rc = ensure_device(ctx, &ctx->work, &ctx->work_elems, nc * ((size_t)Gs * nS + 3 * zv.nm)))) return rc;
    // source grid `which` (0 sfr, 1 xray, 2 + j AGN band bands[j]) of source k, on the device
    // (the AGN histories are re-weighted like the sfr ones, load_reion_bh_grids)
    const rg_grids* sg = src_host ? src_host : g;
    auto src_grid = [&](int k, int which) -> const float* {
      if (which >= 2) {
        const bool hard = bands[which - 2] == 1;
        if (k == 0) return hard ? sg->bh_xray_hard : sg->bh_xray_soft;
        return (hard ? sg->bh_xray_histories_hard : sg->bh_xray_histories_soft) + (size_t)(k - 1) * npad;
      }
      if (k == 0) return which ? sg->xray_luminosity : sg->sfr;
      return (which ? sg->xray_luminosity_histories : sg->sfr_histories) + (size_t)(k - 1) * npad;
    };
    if (src_host && (rc = ensure_device(ctx, &ctx->ts_stage, &ctx->ts_stage_elems, npad * G * used.size()))) return rc;
    auto dev_grid = [&](size_t j, int which) -> const float* {
      return src_host ? ctx->ts_stage + (j * G + which) * npad : src_grid(used[j], which);
    };
    // window rows for the shells (filter() takes BoxSize in Mpc/h and R in Mpc, ComputeTs.c:532)
    // (the sharp-k rows are steps: their cuts are all the passes need)
    if (!sharp) {
      if ((rc = ensure_device(ctx, &ctx->d_radii, &ctx->d_radii_elems, (size_t)nS))) return rc;
      RG_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->d_radii, sh.R.data(), sizeof(double) * nS, cudaMemcpyHostToDevice, st));
      if ((rc = ensure_device(ctx, &ctx->wtab, &ctx->wtab_elems, (size_t)nS * (n2max + 1)))) return rc;
      if ((rc = window_table(ctx, p->BoxSize, ctx->d_radii, nS, p->TsHeatingFilterType, ctx->wtab, n2max, st)))
        return rc;
    }
    auto kzmax = [&](int r) { return std::min(N / 2, (int)std::sqrt((double)cut[r])); };
    std::vector<TsNodeShell> nodes(nS);
    std::memset(nodes.data(), 0, sizeof(TsNodeShell) * nodes.size());

    // Batches of shells, as many as 128 MB of spectra hold (the windows leave a part of each) but at least
    // TS_KB, and TS_KB where combinations pass through the spare slots: the forward transforms of the sources a batch uses first (`used`
    // is in order of first use), then its x and y passes into work[r][g].  From host arrays,
    // each group of sources is copied on the copy stream and its transform waits for the copy,
    // so the copies of later sources overlap the passes of earlier batches.
    size_t next_slot = 0;   // used[0, next_slot) are transformed into spec[slot * G + g]
    const int kb = wide ? TS_KB
                        : std::min(TS_MAXB, std::max(TS_KB, (int)(128.0 * 1024 * 1024 / (8.0 * nc * Gs))));
    // sources per forward launch: host arrays come in small groups, whose copies overlap the passes
    const size_t group = (src_host ? MAXG : fft_forward_group(N)) / G;
    for (int r0 = 0; r0 < nS; r0 += kb) {
      const int cnt = std::min(kb, nS - r0);
      size_t need = next_slot;
      for (int r = r0; r < r0 + cnt; ++r)
        for (int k = 0; k < sh.nsrc; ++k)
          if (sh.coef[(size_t)r * sh.nsrc + k] != 0.f) need = std::max(need, (size_t)slot_of[k] + 1);
      while (next_slot < need) {
        const size_t end = std::min(need, next_slot + group);
        if (src_host) {
          for (size_t j = next_slot; j < end; ++j)
            for (int which = 0; which < G; ++which)
              RG_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->ts_stage + (j * G + which) * npad, src_grid(used[j], which),
                                               sizeof(float) * npad, cudaMemcpyHostToDevice, ctx->copy_stream));
          cudaEvent_t e;
          if ((rc = stage_record(ctx, 4 + next_slot, ctx->copy_stream, &e))) return rc;
          if ((rc = stage_wait(ctx, e, st))) return rc;
        }
        const float* srcs[FWD_MAXG];
        int ng = 0;
        for (size_t j = next_slot; j < end; ++j)
          for (int which = 0; which < G; ++which) srcs[ng++] = dev_grid(j, which);
        if ((rc = fft_forward(ctx, N, srcs, ng, ctx->spec + nc * G * next_slot, nc, 1.0 / std::pow((double)N, 3), st)))
          return rc;
        next_slot = end;
      }
      TsBatch bt;
      std::memset(&bt, 0, sizeof(bt));
      bt.nr = cnt;
      bt.gs = G;
      bt.ng = Gs;
      bt.skip = !xs;
      for (int j = 0; j < cnt; ++j) {
        const int r = r0 + j;
        std::vector<int> ks;
        std::vector<float> cs;
        for (int k = 0; k < sh.nsrc; ++k) {
          const float c = sh.coef[(size_t)r * sh.nsrc + k];
          if (c != 0.f) {
            ks.push_back(slot_of[k]);
            cs.push_back(c);
          }
        }
        if ((int)ks.size() > TS_MAXSRC) {
          // spare slot nused + j holds sum_i cs[i] spec[ks[i]], accumulated in the x pass's order
          const int spare = nused + j;
          if ((rc = ts_combine(ctx, N, ctx->spec, nc, G, ks, cs, spare, st))) return rc;
          ks.assign(1, spare);
          cs.assign(1, 1.f);
        }
        const int nk = (int)ks.size();
        for (int i = 0; i < nk; ++i) {
          bt.ks[j][i] = ks[i];
          bt.cs[j][i] = cs[i];
        }
        bt.nk[j] = nk;
        bt.filtered[j] = r > 0;
        bt.wrow[j] = r;
        bt.cut[j] = cut[r];
        nodes[r].nk = nk;
        nodes[r].filtered = r > 0;
        nodes[r].cut = cut[r];
        std::copy(bt.ks[j], bt.ks[j] + nk, nodes[r].ks);
        std::copy(bt.cs[j], bt.cs[j] + nk, nodes[r].cs);
      }
      if ((rc = ts_xy(ctx, N, ctx->spec, ctx->work + (size_t)r0 * Gs * nc, nc, bt, ctx->wtab, n2max + 1, st)))
        return rc;
    }
    if ((rc = kick())) return rc;
    // the frequency tables, integrated on the side stream during the transforms above
    TsTables tb;
    if ((rc = ts_freq_finish(ctx, p, sh, zp, &tb))) return rc;

    // per-shell coefficients.  evolveInt sums over shells R (XRayHeatingFunctions.c:1379-1432):
    //   heat/ion/lya: dt_dzpp dzpp XRAY_R (1+zpp)^-alpha fi_k(x_e)     (times const_zp later)
    //   star        : SFR_R (1+zp)^2 (1+zpp) sum_lyn dt_dzpp dzpp      (times the conversion)
    // with XRAY_R = xray / pv * 1e40 UL^-3 and SFR_R = max(sfr,0) / pv * (UM/UT) UL^-3 / Msun.
    const double convX = 1.0 / pixel_volume * XRAY_LUMINOSITY_UNIT * std::pow(p->UnitLength_in_cm, -3.);
    const double convS = 1.0 / pixel_volume * (p->UnitMass_in_g / u.UnitTime_in_s) *
                         std::pow(p->UnitLength_in_cm, -3.) / SOLAR_MASS;
    const float zpf = (float)zp;
    const double opzf2 = std::pow((double)(1.0f + zpf), 2);
    std::vector<double> Pd((size_t)nS * 3 * x_int_NXHII), Qd((size_t)nS * 3 * x_int_NXHII), cs(nS);
    double maxk[4] = {0, 0, 0, 0};
    const float* X = ctx->tables.x_int_XHII.data();
    for (int r = 0; r < nS; ++r) {
      const double a = sh.dt_dzpp[r] * sh.dzpp[r];
      const double pw = std::pow(1 + sh.zpp[r], -p->SpecIndexXrayGal);
      for (int kind = 0; kind < 3; ++kind) {
        const std::vector<double>& tb_k = kind == 0 ? tb.heat : kind == 1 ? tb.ion : tb.lya;
        for (int m = 0; m < x_int_NXHII; ++m) {
          const double t_lo = tb_k[(size_t)m * nS + r];
          const double t_hi = m + 1 < x_int_NXHII ? tb_k[(size_t)(m + 1) * nS + r] : t_lo;
          const double slope = m + 1 < x_int_NXHII ? (t_hi - t_lo) / ((double)X[m + 1] - (double)X[m]) : 0.0;
          Pd[((size_t)r * 3 + kind) * x_int_NXHII + m] = a * convX * pw * t_lo;
          Qd[((size_t)r * 3 + kind) * x_int_NXHII + m] = a * convX * pw * slope;
          maxk[kind] = std::max({maxk[kind], std::fabs(a * convX * pw * t_lo), std::fabs(a * convX * pw * t_hi)});
        }
      }
      cs[r] = convS * opzf2 * (1 + sh.zpp[r]) * tb.sum_lyn[r] * a;
      maxk[3] = std::max(maxk[3], std::fabs(cs[r]));
    }
    // AGN bands: XAGN_R = max(bh, 0) 1e10 L_sun / pv UL^-3 (ComputeTs.c:615-630), the band's
    // (1+zpp)^-alpha and tables, and const_zp_AGN / const_zp_GAL so the terms share the
    // galaxies' prefactor in the update kernel (XRayHeatingFunctions.c:1420-1470)
    const double convA = 1e10 * SOLAR_LUM / pixel_volume * std::pow(p->UnitLength_in_cm, -3.0);
    std::vector<double> PAd((size_t)nS * 2 * 3 * x_int_NXHII, 0.0), QAd(PAd.size(), 0.0);
    for (int j = 0; j < nagn; ++j) {
      const int b = bands[j];
      const double alpha_b = b ? p->SpecIndexXrayAGNHard : p->SpecIndexXrayAGNSoft;
      const double ratio = pf.const_zp_prefactor_AGN[b] / pf.const_zp_prefactor_GAL;
      for (int r = 0; r < nS; ++r) {
        const double a = sh.dt_dzpp[r] * sh.dzpp[r] * convA * std::pow(1 + sh.zpp[r], -alpha_b) * ratio;
        for (int kind = 0; kind < 3; ++kind) {
          const std::vector<double>& tb_k = tb.agn[b][kind];
          for (int m = 0; m < x_int_NXHII; ++m) {
            const double t_lo = tb_k[(size_t)m * nS + r];
            const double t_hi = m + 1 < x_int_NXHII ? tb_k[(size_t)(m + 1) * nS + r] : t_lo;
            const double slope = m + 1 < x_int_NXHII ? (t_hi - t_lo) / ((double)X[m + 1] - (double)X[m]) : 0.0;
            const size_t o = (((size_t)r * 2 + j) * 3 + kind) * x_int_NXHII + m;
            PAd[o] = a * t_lo;
            QAd[o] = a * slope;
            maxk[kind] = std::max({maxk[kind], std::fabs(a * t_lo), std::fabs(a * t_hi)});
          }
        }
      }
    }
    // FP32 sums over the shells: scale each sum by a power of two that brings its largest
    // per-shell coefficient near 1 (values of order 1e-30 would lose range in float)
    double scale[4];
    for (int k = 0; k < 4; ++k) {
      scale[k] = pow2_scale(maxk[k]);
      zv.inv_scale[k] = 1.0 / scale[k];
    }
    std::vector<TsShellCoef> hco(nS + 1);
    std::memset(hco.data(), 0, sizeof(TsShellCoef) * hco.size());
    for (int r = 0; r < nS; ++r) {
      for (int kind = 0; kind < 3; ++kind)
        for (int m = 0; m < x_int_NXHII; ++m) {
          hco[r].P[kind][m] = (float)(Pd[((size_t)r * 3 + kind) * x_int_NXHII + m] * scale[kind]);
          hco[r].Q[kind][m] = (float)(Qd[((size_t)r * 3 + kind) * x_int_NXHII + m] * scale[kind]);
        }
      hco[r].cstar = (float)(cs[r] * scale[3]);
      hco[r].kzmax = kzmax(r);
      for (int m = 0; m + 1 < x_int_NXHII; ++m) hco[r].dX[m] = (float)((double)X[m + 1] - (double)X[m]);
      for (int m = 0; m < zv.nm; ++m)
        for (int kind = 0; kind < 3; ++kind)
          nodes[r].f[3 * m + kind] =
              (float)(Pd[((size_t)r * 3 + kind) * x_int_NXHII + zv.m0 + m] * scale[kind]);
      for (int j = 0; j < nagn; ++j)
        for (int kind = 0; kind < 3; ++kind)
          for (int m = 0; m < x_int_NXHII; ++m) {
            const size_t o = (((size_t)r * 2 + j) * 3 + kind) * x_int_NXHII + m;
            hco[r].PA[j][kind][m] = (float)(PAd[o] * scale[kind]);
            hco[r].QA[j][kind][m] = (float)(QAd[o] * scale[kind]);
          }
    }
    // the copies' source lives in the context: nothing here waits for them
    const size_t co_bytes = sizeof(TsShellCoef) * (nS + 1), node_bytes = zv.nm ? sizeof(TsNodeShell) * nS : 0;
    ctx->ts_host.resize(co_bytes + node_bytes);
    std::memcpy(ctx->ts_host.data(), hco.data(), co_bytes);
    if (node_bytes) std::memcpy(ctx->ts_host.data() + co_bytes, nodes.data(), node_bytes);
    RG_CUDA_TRY(ctx, cudaMemcpyAsync(d_co, ctx->ts_host.data(), co_bytes, cudaMemcpyHostToDevice, st));
    zv.nS = nS;
    if (zv.nm) {
      RG_CUDA_TRY(ctx, cudaMemcpyAsync(d_node, ctx->ts_host.data() + co_bytes, node_bytes, cudaMemcpyHostToDevice, st));
      if ((rc = ts_nodes(ctx, N, ctx->spec, ctx->work + (size_t)nS * Gs * nc, nc, G, d_node, nS, zv.nm, ctx->wtab,
                         n2max + 1, st)))
        return rc;
    }
    double planes = 3.0 * zv.nm * (N / 2 + 1);
    for (int r = 0; r < nS; ++r) planes += Gs * (kzmax(r) + 1.0);
    if ((rc = ensure_device(ctx, &ctx->ts_sums, &ctx->ts_sums_elems, n3))) return rc;
    if (nagn && (rc = ensure_device(ctx, &ctx->ts_agn, &ctx->ts_agn_elems, n3))) return rc;
    if ((rc = xy_ctrl_reset(ctx, 0, st))) return rc;   // the error word of the tile waits
    if ((rc = ts_zsum(ctx, N, ctx->work, nc, nagn, d_co, zv, g->x_e_box_prev, ctx->ts_sums,
                      nagn ? ctx->ts_agn : nullptr, planes, st)))
      return rc;
    waits = true;
  }

  TsEvolve e;
  e.zp = zp;
  e.dzp = zp - prev_redshift;
  e.dt_dzp = pf.dt_dzp;
  e.heat_conv = pf.dt_dzp * 2.0 / 3.0 / BOLTZMANN;
  e.growth = pf.growth_factor_zp;
  e.dgrowth = pf.dgrowth_factor_dzp;
  e.const_zp = pf.const_zp_prefactor_GAL;
  // Conversion_factor (XRayHeatingFunctions.c:1331-1332)
  e.conv_star = (SPEED_OF_LIGHT / (4. * M_PI)) / (PROTONMASS / SOLAR_MASS);
  e.no_light = no_light;
  const double4 inv = make_double4(zv.inv_scale[0], zv.inv_scale[1], zv.inv_scale[2], zv.inv_scale[3]);
  prof_begin(ctx, "ts_evolve", st);
  if ((rc = stage_wait(ctx, stg->closing, st))) return rc;
  k_ts_evolve<<<nblk, EV_NT, 0, st>>>(d_hc, par, e, inv, N, no_light ? nullptr : ctx->ts_sums,
                                     (no_light || !nagn) ? nullptr : ctx->ts_agn, g->deltax, g->x_e_box_prev,
                                     g->x_e_box, g->Tk_box, g->TS_box, partials, &d_status->nonconv,
                                     no_light ? nullptr : ctx->xy_ctrl);
  prof_end(ctx, (double)n3 * (16 + 4 + 4 + 4 + 4 + 4 + 4 + 4), st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  return finish(false, nblk);
}

}  // namespace rg
