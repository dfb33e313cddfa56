// Excursion-set step (_find_HII_bubbles, src/core/find_HII_bubbles.c:86-710) on sm_100a.
//
// Per snapshot: one forward r2c of each grid the barrier test reads (deltax, stars, [x_e],
// [effective_bhm]); then the filter radii in batches of KB:
//   x and y passes (rg_hii_xy.cu) into KB x G work grids
//   z pass : per block of rows, for each radius of the batch in order: c2r of the G grids, then the
//            aliasing clamp and the barrier test per cell (k_hii_zr in rg_hii_z.cuh; here the
//            row-buffer form for Pop III sources and the boxes below 64^3, k_hii_z).
// A cell's state over the radii is two bits (ionized this snapshot; z_at_ionization still < 0), kept in
// registers within a batch; between batches k_hii_zr keeps them as two words a thread, k_hii_z as a
// byte per cell.  z_at_ionization and J_21 are written only where a cell first ionizes.  The last radius
// also writes xH, with the sign of "neutral at every radius"; the closing pass (k_hii_close) then takes
// xH and the temperatures to their final values and sums the box averages in FP64.
#include <cuda_runtime.h>
#include <math.h>

#include <cstdio>
#include <algorithm>
#include <cstring>
#include <type_traits>
#include <utility>
#include <vector>

#include "rg_hii_z.cuh"
#include "rg_internal.h"
#include "rg_pass.cuh"

namespace rg {

// ---------------------------------------------------------------------------
// window table W[r][n2], n2 = nx^2 + ny^2 + nz^2, evaluated in double from the closed
// forms of filter() (src/core/reionization.c:3404-3428)

// sharp-k: k R 0.413566994 > 1 zeroes the mode
__device__ __forceinline__ bool sharpk_zero(double delta_k, int n2, double R) {
  const double kR = delta_k * sqrt((double)n2) * R;
  return kR * 0.413566994 > 1.0;
}

__device__ __forceinline__ float window_value(double delta_k, int n2, double R, int ftype) {
  if (ftype == 1) return sharpk_zero(delta_k, n2, R) ? 0.f : 1.f;
  const double kR = delta_k * sqrt((double)n2) * R;
  double w = 1.0;
  if (ftype == 0) {
    if (kR > 1e-4) w = 3.0 * (sin(kR) / (kR * kR * kR) - cos(kR) / (kR * kR));
  } else {
    const double g = kR * 0.643;
    w = exp(-g * g / 2.0);
  }
  return (float)w;
}

// For the sharp-k filter (ftype 1) the row is a step in n2 (kR grows with n2); wcut[r], when
// given, receives the last n2 of the step (written by that entry alone), so
// W[r][n2] == (n2 <= wcut[r]), and the row is not written.
__global__ void k_window_table(float* wtab, int n2max, const double* __restrict__ radii, int nr, double delta_k,
                               int ftype, int* wcut) {
  const int r = blockIdx.y;
  if (r >= nr) return;
  const double R = radii[r];
  for (int n2 = blockIdx.x * blockDim.x + threadIdx.x; n2 <= n2max; n2 += gridDim.x * blockDim.x) {
    const float w = window_value(delta_k, n2, R, ftype);
    if (ftype != 1 || !wcut) {
      wtab[(size_t)r * (n2max + 1) + n2] = w;
    } else if (w == 1.f && (n2 == n2max || sharpk_zero(delta_k, n2 + 1, R))) {
      wcut[r] = n2;
    }
  }
}

// The windows of the radii blockIdx.y on the octant of modes.  The x pass of a radius reads each value
// up to four times per grid, and from a row W[n2] its lanes, at consecutive ny, would gather 32
// different sectors: the planes are read in runs.  One gather fills a mode and its mirror across
// kz = |nx|.  With planes instead of gathers the x/y passes of a 512^3 snapshot (61 radii, 3 grids)
// went from 72.9 to 65.5 ms, of a 256^3 one (42 radii, 2 grids) from 3.69 to 3.35 ms; the planes take
// 2.4 and 0.19 ms.
__global__ void __launch_bounds__(256) k_window_planes(const float* __restrict__ rows, int n2max, int n,
                                                       float* __restrict__ planes) {
  const int h = n / 2 + 1, wp = wplane_pitch(n), kz = blockIdx.x;
  const float* row = rows + (size_t)blockIdx.y * (n2max + 1) + kz * kz;
  float* out = planes + blockIdx.y * wplane_size(n);
  for (int nx = kz + threadIdx.x / 32; nx < h; nx += 8)
    for (int ny = threadIdx.x % 32; ny < h; ny += 32) {
      const float w = __ldg(row + nx * nx + ny * ny);
      out[((size_t)kz * h + nx) * wp + ny] = w;
      out[((size_t)nx * h + kz) * wp + ny] = w;
    }
}

// The plane of one radius by itself (rg_smooth_grid), each value evaluated where it goes: the table and its
// gather are a launch more, about 6 us of a 64^3 call's 60.  smooth_grid, us with window rows gathered in the x/y
// pass, and so: 64^3 60, 55; 128^3 75, 70; 256^3 223, 214; 512^3 1722, 1635.
__global__ void __launch_bounds__(64) k_window_plane(double delta_k, double R, int ftype, int n,
                                                     float* __restrict__ plane) {
  const int h = n / 2 + 1, wp = wplane_pitch(n), kz = blockIdx.x, nx = blockIdx.y;
  if (nx < kz) return;
  for (int ny = threadIdx.x; ny < h; ny += 64) {
    const float w = window_value(delta_k, kz * kz + nx * nx + ny * ny, R, ftype);
    plane[((size_t)kz * h + nx) * wp + ny] = w;
    plane[((size_t)nx * h + kz) * wp + ny] = w;
  }
}

// ---------------------------------------------------------------------------
// temperatures

// ComputeFullyIoinizedTemperature (find_HII_bubbles.c:48-74), with its float/double mix.  The powers
// of constants and of the redshift alone come from the host (HiiConst); the per-cell ones are
// exp(c log(x)), within 1e-13 of x^c for the arguments here (|c log x| < 40), at a third of
// pow's instructions: five pow a cell bounded the closing pass of a mostly ionised box.
__device__ __forceinline__ double pow_pos(double x, double c) { return exp(c * log(x)); }

__device__ __forceinline__ float fully_ionized_T(float z_re, float delta, const HiiConst& k) {
  const float z = k.redshift;
  float result, delta_re;
  if (fabs((double)(z - z_re)) < 1e-4) {
    result = 1.f;
  } else {
    const double ratio = (1.0 + (double)z) / (1.0 + (double)z_re);
    delta_re = (float)((double)delta * (1.0 + (double)z) / (1.0 + (double)z_re));
    if (delta_re <= -1.f) delta_re = (float)(-1.0 + (double)ABS_TOL);
    if (delta <= -1.f) delta = (float)(-1.0 + (double)ABS_TOL);
    result = (float)pow_pos((1.0 + (double)delta) / (1.0 + (double)delta_re), 1.1333);
    result = (float)((double)result * pow_pos(ratio, 3.4));
    const double b = (1.0 + (double)z_re) / 7.1;
    result *= expf((float)(k.z_25 - b * b * sqrt(b)));
  }
  result = (float)((double)result * k.t_17);
  result = (float)((double)result + k.z_17 * (double)(1.f + delta));
  return (float)pow_pos((double)result, 0.5882);
}

// Block sum of K doubles per thread into out[0..K), deterministic order.
template <int NTH, int K>
__device__ __forceinline__ void block_sum(double (&acc)[K], double* out) {
  if constexpr (NTH % 32 == 0) {
    __shared__ double s_red[NTH / 32][K];
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
      for (int w = 0; w < NTH / 32; ++w) v += s_red[w][threadIdx.x];
      out[threadIdx.x] = v;
    }
  } else {
    __shared__ double s_red[NTH][K];
#pragma unroll
    for (int i = 0; i < K; ++i) s_red[threadIdx.x][i] = acc[i];
    __syncthreads();
    if (threadIdx.x < K) {
      double v = 0.0;
      for (int w = 0; w < NTH; ++w) v += s_red[w][threadIdx.x];
      out[threadIdx.x] = v;
    }
  }
}

// ---------------------------------------------------------------------------
// closing pass (find_HII_bubbles.c:577-645): one cell a thread in memory order, so every access is
// coalesced (in the z pass, whose threads hold a few cells of many rows, it took 5 ms of a 512^3
// snapshot).  In: xH with the sign of "neutral at every radius" (the z pass).  A partly ionised
// cell's temperature, ComputePartiallyIoinizedTemperature of the neutral gas's T at residual xH 1,
// is that T: Tk_box with the spin temperature, else the adiabatic T; the floor is the same T.
constexpr int CLOSE_NT = 256;
struct HiiCloseUnits {   // snapshots of a launch (blockIdx.y)
  HiiConst c[HII_ZU];
  HiiState s[HII_ZU];
};

template <int N>
__global__ void __launch_bounds__(CLOSE_NT) k_hii_close(const __grid_constant__ HiiCloseUnits us,
                                                        double* __restrict__ partials) {
  const HiiConst& c = us.c[blockIdx.y];
  const HiiState& s = us.s[blockIdx.y];
  constexpr int PADW = 2 * (N / 2 + 1);
  const size_t n3 = (size_t)N * N * N;
  double acc[HII_NSUM];
#pragma unroll
  for (int k = 0; k < HII_NSUM; ++k) acc[k] = 0.0;
  for (size_t ir = (size_t)blockIdx.x * CLOSE_NT + threadIdx.x; ir < n3; ir += (size_t)gridDim.x * CLOSE_NT) {
    const size_t ip = ir / N * PADW + ir % N;
    const float xs = s.xH[ir], du = s.deltax_unf[ip], zin = s.z_in[ir], told = s.temp[ir], ws = s.wsfr[ip];
    const bool neutral = signbit(xs);
    const float xH = fabsf(xs);
    const float tn = c.spin ? s.Tk_box[ir] : (float)((double)c.TK * (1.0 + (double)(c.cT_ad * du)));
    float temp = neutral ? tn : told;
    if (xH < REL_TOL && zin > 0.f) temp = fully_ionized_T(zin, du, c);
    if (temp < tn) temp = tn;
    if (neutral) s.xH[ir] = xH;
    s.temp[ir] = temp;
    const double domu = 1.0 + (double)du;
    acc[0] += (double)xH;
    // acc[1] and acc[6]: r_bubble is written only on the recombination branch
    // (find_HII_bubbles.c:490-508); its sums come from k_hii_recomb.
    acc[2] += (double)ws;
    if (s.bhar != nullptr) acc[3] += (double)s.bhar[ip];
    if (s.wsfrIII != nullptr) acc[9] += (double)s.wsfrIII[ip];
    acc[4] += (double)temp;
    acc[5] += (double)xH * domu;
    acc[7] += (double)temp * domu;
    acc[8] += domu;
  }
  block_sum<CLOSE_NT, HII_NSUM>(acc, partials + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * HII_NSUM);
}

template <int N>
int launch_hii_close(rg_context* ctx, const HiiCloseUnits& us, int nu, double* partials, int nblocks,
                     cudaStream_t st) {
  prof_begin(ctx, "hii_close", st);
  k_hii_close<N><<<dim3(nblocks, nu), CLOSE_NT, 0, st>>>(us, partials);
  // xH, deltax, z_at_ionization, temperature, weighted_sfr (and Tk_box, ...) read, xH and temperature written
  prof_end(ctx, nu * 4.0 * N * N * N * (7 + us.c[0].spin + (us.s[0].bhar != nullptr) + (us.s[0].wsfrIII != nullptr)),
           st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  return RG_OK;
}

// ---------------------------------------------------------------------------
// the z pass with Pop III sources, and of the boxes below 64^3: up to 9 grids a radius, in row buffers
//
// Shared-memory plan: ZB tile buffers of TB complex each; the buffer of the unit
// being transformed is also its FFT exchange buffer (the tile is consumed by the first stage).
// Two buffers let the next grid's tile arrive while this one is transformed.  At 512^3 one buffer
// brings a block to 72 KB and the SM to three blocks instead (46.0 -> 44.0 ms over 7 batches of 8
// radii and 3 grids).
template <int N>
struct HiiZ {
  static constexpr int NTH = Cfg<N>::T * Cfg<N>::QZ;
  static constexpr bool WIDE = N == 512;
  static constexpr int ZB = WIDE ? 1 : 2;
  static constexpr int TB = round_up(cmax((int)ztile_elems<N>(), line_buf<N, Cfg<N>::QZ>()), 2);
  static constexpr int MINB = WIDE ? 3 : RG_MINB(NTH);
  static constexpr size_t smem(int ng) {
    return sizeof(cf) * (size_t)N + sizeof(float) * (size_t)round_up(ng * 2 * Cfg<N>::QZ * Cfg<N>::RT_PITCH, 4) +
           sizeof(cf) * (size_t)ZB * TB;
  }
};

// z pass of a batch.
// Grids in rt: 0 deltax, 1 stars, then x_e (spin temperature), then effective_bhm (BH), then
// starsIII (Pop III), then with recombinations N_rec, weighted_sfr, effective_bhar (BH) and
// weighted_sfrIII (Pop III); bt.ng of them.
//
// NG: the number of grids (2 to 4) without recombinations or Pop III, so that the loop over them and the
// test compile without the other grids' branches; 0: any count, from bt.  FINAL: the batch ends with the
// snapshot's last radius (as in k_hii_zr).  With both known only at run time the pass of a small box took
// about twice as long: 24^3, 34 radii of 2 grids, 483 us against 209; 48^3, 41 radii, 770 against 375;
// 128^3 with Pop III sources 1.90 ms a call against 1.84.
template <int N, int NG, bool FINAL>
__global__ void __launch_bounds__(Cfg<N>::T* Cfg<N>::QZ, (HiiZ<N>::MINB))
    k_hii_z(const cf* __restrict__ work, size_t stride, const cf* __restrict__ g_tw, HiiBatch bt, HiiBatchIII b3,
            HiiConst c, HiiState s) {
  constexpr int T = Cfg<N>::T, Q = Cfg<N>::QZ, NTH = T * Q, ROWS = 2 * Q, RP = Cfg<N>::RT_PITCH;
  constexpr int PADW = 2 * (N / 2 + 1);
  constexpr int IT = ROWS * N / NTH;   // cells per thread
  constexpr int W = (IT + 31) / 32;    // bit words per thread
  static_assert(ROWS * N % NTH == 0, "whole rows per block");
  extern __shared__ __align__(16) unsigned char smem_raw[];  // 16-byte aligned for cp.async
  cf* smem = reinterpret_cast<cf*>(smem_raw);
  constexpr int ZB = HiiZ<N>::ZB, TB = HiiZ<N>::TB;
  cf* s_tw = smem;
  float* rt = reinterpret_cast<float*>(smem + N);
  // ZB shared tiles (with two, grid u + 1 is copied while grid u is transformed); the tile of
  // unit u is the exchange buffer of its transform
  // (after the row buffers of the grids there are)
  const int ng = NG ? NG : bt.ng;
  cf* tiles = reinterpret_cast<cf*>(rt + round_up(ng * ROWS * RP, 4));
  const int x = blockIdx.y, y0 = blockIdx.x * ROWS;
  load_twiddles<N>(s_tw, g_tw);

  // per-cell state bits: A = z_at_ionization still < 0, I = ionized at a radius of this snapshot.
  // Cell it of this thread is block cell threadIdx.x + it * NTH, bit it % 32 of word it / 32;
  // between batches the state is one byte per cell (s.state, bit 0 = A, bit 1 = I).
  uint32_t A[W], I[W];
#pragma unroll
  for (int w = 0; w < W; ++w) {
    uint32_t a = 0u, iv = 0u;
    const int nb = IT - 32 * w < 32 ? IT - 32 * w : 32;
#pragma unroll 8
    for (int bb = 0; bb < nb; ++bb) {
      const int i = threadIdx.x + (32 * w + bb) * NTH;
      const size_t ir = ((size_t)x * N + y0 + i / N) * N + i % N;
      if (bt.first) {
        if (s.z_in[ir] < 0.f) a |= 1u << bb;
      } else {
        const uint32_t v = s.state[ir];
        a |= (v & 1u) << bb;
        iv |= ((v >> 1) & 1u) << bb;
      }
    }
    A[w] = a;
    I[w] = iv;
  }
  const bool rec = NG == 0 && c.rec, mini = NG == 0 && c.mini;
  int gi = 2;
  const int gx = c.spin ? gi++ : -1;
  const int gb = c.bh ? gi++ : -1;
  const int gm = mini ? gi++ : -1;                 // starsIII
  const int gn = rec ? gi++ : -1;                  // N_rec
  const int gw = rec ? gi++ : -1;                  // weighted_sfr
  const int gr = rec && c.bh ? gi++ : -1;          // effective_bhar
  const int gw3 = rec && mini ? gi++ : -1;         // weighted_sfrIII

  const int nunits = bt.nr * ng;   // (radius, grid) pairs, unit u = r * ng + g
  ztile_issue<N, Q>(tiles, work, x, y0, NTH);
  cp_async_commit();
  const int q = threadIdx.x % Q, tq = threadIdx.x / Q;
  for (int r = 0; r < bt.nr; ++r) {
    __syncthreads();  // rt of the previous radius is consumed
#pragma unroll 1
    for (int g = 0; g < ng; ++g) {
      const int u = r * ng + g;
      cf* tile = tiles + (ZB == 2 ? (u & 1) : 0) * TB;
      if constexpr (ZB == 2) {
        if (u + 1 < nunits) ztile_issue<N, Q>(tiles + ((u + 1) & 1) * TB, work + (size_t)(u + 1) * stride, x, y0, NTH);
        cp_async_commit();
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncthreads();  // unit u's tile is complete for every thread
      float* r0 = rt + (size_t)(g * ROWS + 2 * q) * RP;
      line_fft<N, true>(
          tq, tile, s_tw, [&](int p, int) { return ztile_c2r_input<N, Q>(tile, q, p); },
          [&](int p) { return line_addr<N, Q>(p, q); },
          [&](int p, cf v) {
            r0[p] = v.x;
            r0[RP + p] = v.y;
          });
      __syncthreads();  // the tile is consumed before it is refilled; rt row is written
      if constexpr (ZB == 1) {
        if (u + 1 < nunits) ztile_issue<N, Q>(tiles, work + (size_t)(u + 1) * stride, x, y0, NTH);
        cp_async_commit();
      }
    }
    const bool last = FINAL && r == bt.nr - 1;
    const double pref = bt.fcoll_pref[r];
#pragma unroll
    for (int w = 0; w < W; ++w) {
      uint32_t a = A[w], iw = I[w];
      const int nb = IT - 32 * w < 32 ? IT - 32 * w : 32;
#pragma unroll 4
      for (int bb = 0; bb < nb; ++bb) {
        const int i = threadIdx.x + (32 * w + bb) * NTH;
        const int z = i % N, row = i / N;
        const uint32_t bit = 1u << bb;
        const float dx = fmaxf(rt[row * RP + z], -1.f + REL_TOL);
        float st = fmaxf(rt[(ROWS + row) * RP + z], 0.f);
        if (st < ABS_TOL) st = 0.f;
        float xe = 0.f, bhm = 0.f;
        if (gx >= 0) {
          xe = fmaxf(rt[(gx * ROWS + row) * RP + z], 0.f);
          if (xe < ABS_TOL) xe = 0.f;
          xe = fminf(xe, 0.999f);
        }
        if (gb >= 0) {
          bhm = fmaxf(rt[(gb * ROWS + row) * RP + z], 0.f);
          if (bhm < ABS_TOL) bhm = 0.f;
        }
        float stIII = 0.f;
        if (gm >= 0) {
          stIII = fmaxf(rt[(gm * ROWS + row) * RP + z], 0.f);
          if (stIII < ABS_TOL) stIII = 0.f;
        }
        float nrec = 0.f;
        if (gn >= 0) {
          nrec = fmaxf(rt[(gn * ROWS + row) * RP + z], 0.f);
          if (nrec < ABS_TOL) nrec = 0.f;
        }
        const double dom = 1.0 + (double)dx;  // >= 1e-5 after the clamp
        const double nf = c.spin ? 1.0 - (double)xe : 1.0;
        const double rec = gn >= 0 ? (double)nrec / dom : 0.0;
        // (f_bh + f_stars) * prefactor > nf (1 + rec) with f = grid / dom, tested with both
        // sides times dom: the two forms differ only within a few FP64 ulps of the barrier
        const double num = c.bh ? (double)bhm + (double)st : (double)st;
        const double prefIII = gm >= 0 ? b3.fcoll_pref[r] : 0.0;
        const double lhs_dom = gm >= 0 ? num * pref + (double)stIII * prefIII : num * pref;
        const bool ion = lhs_dom > nf * (1.0 + rec) * dom;
        float xH = (iw & bit) ? 0.f : 1.f;   // so far: 0 once ionized at a radius, else 1
        const size_t cellrow = (size_t)x * N + y0 + row;
        const size_t ir = cellrow * N + z;
        if (ion) {
          if (gn >= 0 && !(iw & bit)) {
            // first crossing of the snapshot (find_HII_bubbles.c:488-508)
            float wsf = fmaxf(rt[(gw * ROWS + row) * RP + z], 0.f);
            if (wsf < ABS_TOL) wsf = 0.f;
            float G = __fmul_rn(wsf, bt.G_pref[r]);
            if (gw3 >= 0) {
              float w3 = fmaxf(rt[(gw3 * ROWS + row) * RP + z], 0.f);
              if (w3 < ABS_TOL) w3 = 0.f;
              G = __fadd_rn(G, __fmul_rn(w3, b3.G_pref[r]));
            }
            if (gr >= 0) {
              float bhr = fmaxf(rt[(gr * ROWS + row) * RP + z], 0.f);
              if (bhr < ABS_TOL) bhr = 0.f;
              G = __fadd_rn(G, __fmul_rn(bhr, bt.G_pref_bh[r]));
            }
            s.Gamma12[ir] = G;
            s.r_bubble[ir] = bt.R[r];
            if (c.uvb == 2) {
              float j = __fmul_rn(st, bt.J_aux[r]);
              if (gm >= 0) j = __fadd_rn(j, __fmul_rn(stIII, b3.J_aux[r]));
              if (c.bh) j = __fadd_rn(j, __fmul_rn(bhm, bt.J_aux_bh[r]));
              s.J21[ir] = j;
            }
          }
          xH = 0.f;
          iw |= bit;
        } else if (last && xH > REL_TOL) {
          // partially ionized: xH = nf - f_coll prefactor
          const double fcs = (double)st / dom;
          const double fbh = c.bh ? (double)bhm / dom : 0.0;
          const double lhs = (fbh + fcs) * pref;
          float v = (float)(nf - lhs);
          if (gm >= 0) v -= (float)((double)stIII / dom * prefIII);   // a float subtraction in the C
          xH = v < 0.f ? 0.f : (v > 1.f ? 1.f : v);
        }
        if (xH < REL_TOL && (a & bit)) {
          // new ionization (find_HII_bubbles.c:531-543)
          a &= ~bit;
          s.z_in[ir] = c.redshift;
          if (c.uvb == 1) {
            float j = st * bt.J_aux[r];
            if (gm >= 0) j = __fadd_rn(j, __fmul_rn(stIII, b3.J_aux[r]));
            if (c.bh) j += bhm * bt.J_aux_bh[r];
            s.J21[ir] = j;
          }
        }
        if (last) s.xH[ir] = (iw & bit) ? 0.f : -xH;   // the sign: neutral at every radius (k_hii_close)
      }
      A[w] = a;
      I[w] = iw;
    }
  }

  if constexpr (!FINAL) {
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const int nb = IT - 32 * w < 32 ? IT - 32 * w : 32;
#pragma unroll 8
      for (int bb = 0; bb < nb; ++bb) {
        const int i = threadIdx.x + (32 * w + bb) * NTH;
        const size_t ir = ((size_t)x * N + y0 + i / N) * N + i % N;
        s.state[ir] = (uint8_t)(((A[w] >> bb) & 1u) | (((I[w] >> bb) & 1u) << 1));
      }
    }
  }
}

// deterministic second stage: block (i, u) sums sum i of the per-block partials of set u in a fixed
// order (one block for all the sums took 11 to 28 us)
__global__ void __launch_bounds__(256) k_reduce_partials(const double* __restrict__ partials, int nblocks, int nsum,
                                                         double* out, size_t set_pitch, int out_pitch) {
  __shared__ double sh[256];
  const int i = blockIdx.x;
  partials += blockIdx.y * set_pitch;
  double v = 0.0;
  for (int b = threadIdx.x; b < nblocks; b += 256) v += partials[(size_t)b * nsum + i];
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[blockIdx.y * out_pitch + i] = sh[0];
}

// ---------------------------------------------------------------------------
// launchers

// ---------------------------------------------------------------------------
// recombinations in the closing pass (find_HII_bubbles.c:612-644)

struct RecConst {
  double redshift;     // ZZ[snapshot]
  double hubble_h;
  float fabs_dtdz;     // |dt/dz| / h at the snapshot, float as in the reference
  float zstep;         // ZZ[snapshot - 1] - ZZ[snapshot] (0 at snapshot 0)
  int temp_dep;        // Flag_TemperatureDependentRec
};

struct RecState {
  const float* xH;
  const float* temp;         // temp_kinetic_all_gas after the closing pass
  const float* deltax_unf;   // padded
  const float* r_bubble;
  const float* Gamma12;
  float* N_rec;              // padded
  float* residual_xH;
  float* clumping_factor;
  float* t_resp;
};

constexpr int REC_NSUM = 10;   // r_bubble, Gamma12, N_rec, residual_xH, clumping: volume and mass
constexpr int REC_NT = 256;

// splined_recombination (recombinations.c:35-84): the (z, T) row by rounding to the nearest
// sample, then the natural cubic spline in ln Gamma12 of that row.  The sample spacings are
// the float constants of recombinations.h:17-34.
__device__ void splined_recombination(const RecTables& t, double z_eff, double gamma12, double temp, double* rate,
                                      double* rnh, double* cf) {
  int z_ct = (int)((z_eff - (double)0.0f) / (double)0.2f + 0.5);
  int t_ct = (int)((log10(temp) - (double)2.0f) / (double)0.03f + 0.5);
  double lng = log(gamma12);
  if (z_ct < 0)
    z_ct = 0;
  else if (z_ct >= t.nz)
    z_ct = t.nz - 1;
  if (t_ct < 0 || !(lng >= t.lng_lo)) {
    *rate = 0.0;
    *rnh = 1e4;
    *cf = 1.0;
    return;
  }
  if (t_ct >= t.nt) t_ct = t.nt - 1;
  if (lng >= t.lng_hi) lng = t.lng_hi - 1e-7;   // FRACT_FLOAT_ERR
  // interval lo with knots[lo] <= lng < knots[lo + 1]
  int lo = 0, hi = t.ng - 1;
  while (hi > lo + 1) {
    const int mid = (lo + hi) >> 1;
    if (t.knots[mid] > lng)
      hi = mid;
    else
      lo = mid;
  }
  const double xlo = t.knots[lo];
  const double h = t.knots[lo + 1] - xlo, dx = lng - xlo;
  const size_t rows = (size_t)t.nz * t.nt;
  const size_t row = (size_t)z_ct * t.nt + t_ct;
  double v[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const size_t o = ((size_t)k * rows + row) * t.ng + lo;
    const double yl = t.y[o], yh = t.y[o + 1], cl = t.c[o], ch = t.c[o + 1];
    const double b = (yh - yl) / h - h * (ch + 2.0 * cl) / 3.0;
    const double d = (ch - cl) / (3.0 * h);
    v[k] = yl + dx * (b + dx * (cl + dx * d));
  }
  *rate = exp(v[0]);
  *cf = v[1];
  *rnh = exp(v[2]);
}

template <int N>
__global__ void __launch_bounds__(REC_NT) k_hii_recomb(RecTables tab, RecConst c, RecState s, double* partials) {
  constexpr int PADW = 2 * (N / 2 + 1);
  const size_t n3 = (size_t)N * N * N;
  double acc[REC_NSUM];
#pragma unroll
  for (int k = 0; k < REC_NSUM; ++k) acc[k] = 0.0;
  for (size_t ir = (size_t)blockIdx.x * REC_NT + threadIdx.x; ir < n3; ir += (size_t)gridDim.x * REC_NT) {
    const size_t ip = ir / N * PADW + ir % N;
    const float xHf = s.xH[ir];
    const double dom = 1.0 + (double)s.deltax_unf[ip];
    const double z_eff = (1.0 + c.redshift) * pow(dom, 1.0 / 3.0) - 1.0;
    const double temp = c.temp_dep ? (double)s.temp[ir] : 1e4;
    const float G = s.Gamma12[ir];
    const double gh = __dmul_rn(__dmul_rn((double)G, c.hubble_h), c.hubble_h);
    double rate, rnh, cf;
    splined_recombination(tab, z_eff, gh, temp, &rate, &rnh, &cf);
    // N_rec += (float)rate * fabs_dtdz * zstep * (1 - xH): a float product, widened
    const float f = __fmul_rn(__fmul_rn((float)rate, c.fabs_dtdz), c.zstep);
    const float nrec = (float)__dadd_rn((double)s.N_rec[ip], __dmul_rn((double)f, 1.0 - (double)xHf));
    s.N_rec[ip] = nrec;
    const float rnhf = (float)rnh, cff = (float)cf;
    s.residual_xH[ir] = rnhf;
    s.clumping_factor[ir] = cff;
    // t_resp = 1 / (Gamma + rate) in Myr, stored as float first (find_HII_bubbles.c:630-635)
    float tr = (float)__dadd_rn(__dmul_rn(gh, 1e-12), rate);
    tr = tr > 0.f ? (float)(1.0 / (double)tr / SEC_PER_MEGAYEAR) : 1e30f;
    s.t_resp[ir] = tr;
    const double rb = (double)s.r_bubble[ir];
    acc[0] += rb;
    acc[1] += rb * dom;
    acc[2] += (double)G;
    acc[3] += (double)G * dom;
    acc[4] += (double)nrec;
    acc[5] += (double)nrec * dom;
    acc[6] += (double)rnhf;
    acc[7] += (double)rnhf * dom;
    acc[8] += (double)cff;
    acc[9] += (double)cff * dom;
  }
  block_sum<REC_NT, REC_NSUM>(acc, partials + (size_t)blockIdx.x * REC_NSUM);
}

template <int N>
int launch_hii_recomb(rg_context* ctx, const RecTables& tab, const RecConst& c, const RecState& s, double* partials,
                      int nblocks, cudaStream_t st) {
  prof_begin(ctx, "hii_recomb", st);
  k_hii_recomb<N><<<nblocks, REC_NT, 0, st>>>(tab, c, s, partials);
  // xH, temperature, deltax, r_bubble, Gamma12 read; N_rec read and written; three outputs
  prof_end(ctx, 40.0 * (double)N * N * N, st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  return RG_OK;
}

template <typename K>
static cudaError_t prep(K kernel, size_t smem) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

// grids k_hii_z can hold at this size: the most, up to 9, whose row buffers fit the
// 227 KB of shared memory a block may use (7 at 384^3, 8 at 192^3)
template <int N>
constexpr int hii_ngx() {
  int ng = 9;
  while (ng > 4 && HiiZ<N>::smem(ng) > 227 * 1024) --ng;
  return ng;
}

template <int N, int NG>
int launch_hii_zrow(rg_context* ctx, const cf* work, size_t stride, const HiiZUnit& u, const HiiBatchIII& b3,
                    cudaStream_t st) {
  const cf* tw;
  int rc = twiddles_for(ctx, N, &tw);
  if (rc) return rc;
  using C = Cfg<N>;
  const HiiBatch& bt = u.bt;
  constexpr int NGX = NG ? NG : hii_ngx<N>();
  if (bt.ng > NGX)
    return set_error(ctx, RG_EUNSUPPORTED,
                     "this combination of grids (recombinations, Pop III, BH feedback, spin temperature) needs "
                     "more row buffers than one z pass holds at this ReionGridDim");
  static_assert(HiiZ<N>::smem(NGX) <= 227 * 1024, "z pass shared memory above the per-block limit");
  // the shared memory of the grids there are, not of the maximum
  const size_t sm = HiiZ<N>::smem(bt.ng);
  auto kern = bt.last ? k_hii_z<N, NG, true> : k_hii_z<N, NG, false>;
  RG_CUDA_TRY(ctx, prep(kern, HiiZ<N>::smem(NGX)));
  const dim3 grid(N / (2 * C::QZ), N);
  // algorithmic bytes: the Hermitian halves of the grids per radius, z_at_ionization on the
  // first batch, xH at the end
  const double n3 = (double)N * N * N, nzc = (double)C::NZ * N * N;
  prof_begin(ctx, bt.last ? "inv_z_c2r_test_final" : "inv_z_c2r_test", st);
  kern<<<grid, C::T * C::QZ, sm, st>>>(work, stride, tw, bt, b3, u.c, u.s);
  prof_end(ctx, bt.nr * bt.ng * 8.0 * nzc + (bt.first || bt.last ? 4.0 * n3 : 2.0 * n3), st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  return RG_OK;
}

// the z pass of one batch for nu snapshots (one with Pop III sources: b3), whose windowed spectra lie
// one after another in work
template <int N>
int launch_hii_z(rg_context* ctx, const cf* work, size_t stride, int ng, int nu, const HiiZUnits& us,
                 const HiiBatchIII& b3, cudaStream_t st) {
  const HiiConst& c = us.u[0].c;
  auto row = [&](auto ngc, int k) {
    return launch_hii_zrow<N, decltype(ngc)::value>(ctx, work + (size_t)k * us.u[k].bt.nr * ng * stride, stride,
                                                    us.u[k], b3, st);
  };
  if constexpr (HiiZR<N>::USED) {
    if (!c.mini) return launch_hii_zr<N>(ctx, work, nu, us, st);
  }
  for (int k = 0; k < nu; ++k) {
    int rc;
    if constexpr (HiiZR<N>::USED) {
      rc = row(std::integral_constant<int, 0>{}, k);
    } else {
      rc = c.mini || c.rec ? row(std::integral_constant<int, 0>{}, k)
           : ng == 2       ? row(std::integral_constant<int, 2>{}, k)
           : ng == 3       ? row(std::integral_constant<int, 3>{}, k)
                           : row(std::integral_constant<int, 4>{}, k);
    }
    if (rc) return rc;
  }
  return RG_OK;
}

template <int N>
int launch_debug_inverse(rg_context* ctx, const cf* spec, cf* work, const float* wplane, float* out, cudaStream_t st) {
  const size_t stride = (size_t)Cfg<N>::NZ * N * N;
  int rc = xy_ctrl_reset(ctx, Cfg<N>::NZ, st);
  if (rc) return rc;
  rc = inverse_xy(ctx, N, spec, 1, 1, work, stride, 1, wplane, wplane ? -1 : 0, st, nullptr);
  if (rc) return rc;
  const cf* tw;
  if ((rc = twiddles_for(ctx, N, &tw))) return rc;
  using C = Cfg<N>;
  const size_t sm = zfront_smem_bytes<N>(1);
  RG_CUDA_TRY(ctx, prep(k_inv_z_padded<N>, sm));
  k_inv_z_padded<N><<<dim3(N / (2 * C::QZ), N), C::T * C::QZ, sm, st>>>(work, tw, out);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  return RG_OK;
}

static int hii_z(rg_context* ctx, int n, const cf* work, size_t stride, int ng, int nu, const HiiZUnits& us,
                 const HiiBatchIII& b3, cudaStream_t st) {
  RG_DISPATCH_N(n, launch_hii_z<NN>(ctx, work, stride, ng, nu, us, b3, st));
}

// snapshots one z launch takes at this size
static int hii_z_units(int n) { return n <= 128 ? HII_ZU : 1; }

// the closing passes of nu snapshots; snapshot u's partial sums at partials + u nblocks HII_NSUM
static int hii_close(rg_context* ctx, int n, const HiiConst* c, const HiiState* s, int nu, double* partials,
                     int nblocks, cudaStream_t st) {
  for (int u0 = 0; u0 < nu; u0 += HII_ZU) {
    const int cu = std::min(HII_ZU, nu - u0);
    HiiCloseUnits us;
    std::copy(c + u0, c + u0 + cu, us.c);
    std::copy(s + u0, s + u0 + cu, us.s);
    double* p = partials + (size_t)u0 * nblocks * HII_NSUM;
    auto go = [&]() -> int { RG_DISPATCH_N(n, launch_hii_close<NN>(ctx, us, cu, p, nblocks, st)); };
    const int rc = go();
    if (rc) return rc;
  }
  return RG_OK;
}

static int hii_recomb(rg_context* ctx, int n, const RecTables& tab, const RecConst& c, const RecState& s,
                      double* partials, int nblocks, cudaStream_t st) {
  RG_DISPATCH_N(n, launch_hii_recomb<NN>(ctx, tab, c, s, partials, nblocks, st));
}

int window_table(rg_context* ctx, double box, const double* d_radii, int nr, int ftype, float* d_wtab, int n2max,
                 cudaStream_t st, int* d_wcut) {
  const double delta_k = 2.0 * M_PI / box;
  const int bx = (n2max + 1 + 255) / 256;
  if (ftype != 1) d_wcut = nullptr;
  prof_begin(ctx, "window_table", st);
  k_window_table<<<dim3(bx < 1024 ? bx : 1024, nr), 256, 0, st>>>(d_wtab, n2max, d_radii, nr, delta_k, ftype, d_wcut);
  prof_end(ctx, 4.0 * (n2max + 1) * nr, st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  return RG_OK;
}

int window_planes(rg_context* ctx, int n, const float* wrows, int nr, float* planes, cudaStream_t st) {
  const int n2max = 3 * (n / 2) * (n / 2);
  prof_begin(ctx, "window_planes", st);
  k_window_planes<<<dim3(n / 2 + 1, nr), 256, 0, st>>>(wrows, n2max, n, planes);
  prof_end(ctx, 4.0 * wplane_size(n) * nr, st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  return RG_OK;
}

int reduce_partials(rg_context* ctx, const double* partials, int nblocks, int nsum, double* d_out, cudaStream_t st,
                    int sets, size_t set_pitch, int out_pitch) {
  prof_begin(ctx, "reduce_partials", st);
  k_reduce_partials<<<dim3(nsum, sets), 256, 0, st>>>(partials, nblocks, nsum, d_out, set_pitch, out_pitch);
  prof_end(ctx, 8.0 * nblocks * nsum * sets, st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  return RG_OK;
}

int xy_ctrl_reset(rg_context* ctx, size_t max_jobs, cudaStream_t st) {
  int rc = ensure_device(ctx, &ctx->xy_ctrl, &ctx->xy_ctrl_elems, max_jobs + 2);
  if (rc) return rc;
  RG_CUDA_TRY(ctx, cudaMemsetAsync(ctx->xy_ctrl, 0, sizeof(uint32_t), st));
  return RG_OK;
}

int xy_ctrl_fetch(rg_context* ctx, cudaStream_t st) {
  std::memset(ctx->h_sums + 63, 0, sizeof(double));
  if (ctx->xy_ctrl)
    RG_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_sums + 63, ctx->xy_ctrl, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  return RG_OK;
}

int xy_ctrl_result(rg_context* ctx) {
  uint32_t err;
  std::memcpy(&err, ctx->h_sums + 63, sizeof(err));
  if (err)
    return set_error(ctx, RG_ETIMEDOUT,
                     "a bounded device wait ran out (the fused x/y pass's wait for a plane, or a tensor tile's)");
  return RG_OK;
}

int xy_ctrl_check(rg_context* ctx, cudaStream_t st) {
  int rc = xy_ctrl_fetch(ctx, st);
  if (rc) return rc;
  RG_CUDA_TRY(ctx, cudaStreamSynchronize(st));
  return xy_ctrl_result(ctx);
}

// ---------------------------------------------------------------------------
// the snapshot

// per-snapshot constants of the z passes
static int hii_const(rg_context* ctx, const rg_params* p, double redshift, HiiConst* c) {
  const double tk_d = T_RECFAST(ctx->tables, (float)redshift);
  if (tk_d < 0) return set_error(ctx, RG_ETABLE, "T_RECFAST called beyond its table");
  c->redshift = (float)redshift;
  c->TK = (float)tk_d;
  c->cT_ad = cT_approx((float)redshift);
  c->uvb = p->ReionUVBFlag;
  c->spin = p->Flag_IncludeSpinTemp != 0;
  c->bh = p->Flag_BHFeedback != 0;
  c->rec = p->Flag_IncludeRecombinations != 0;
  c->mini = p->UseMiniHalos != 0;
  const double opz = 1.0 + (double)c->redshift;
  c->t_17 = std::pow(T_RE, 1.7);
  c->z_17 = std::pow(1e4 * (opz / 4.0), 1.7);
  c->z_25 = std::pow(opz / 7.1, 2.5);
  return RG_OK;
}

// the per-radius prefactors of radii [r0, r0 + cnt) (find_HII_bubbles.c:430-450)
static void hii_batch_radii(const rg_params* p, double redshift, const std::vector<std::pair<double, bool>>& sched,
                            int r0, int cnt, int ntest, HiiBatch* bt, HiiBatchIII* b3) {
  const int N = p->ReionGridDim;
  const double pixel_volume = std::pow(p->BoxSize / (double)N, 3);
  const Units u = make_units(p);
  const double sfr_timescale = p->ReionSfrTimescale * hubble_time_at(p, redshift);
  std::memset(bt, 0, sizeof(*bt));
  bt->nr = cnt;
  bt->first = (r0 == 0);
  bt->last = (r0 + cnt == (int)sched.size());
  bt->ng = ntest;
  for (int k = 0; k < cnt; ++k) {
    const double R = sched[r0 + k].first;
    const double M_mean = rtom(p, R);
    double Gamma_R_prefactor = (1.0 + redshift) * (1.0 + redshift) * R * p->UnitLength_in_cm / pixel_volume *
                               std::pow(p->UnitLength_in_cm, -3.);
    Gamma_R_prefactor *= (p->UnitMass_in_g / u.UnitTime_in_s) / PROTONMASS * p->ReionNionPhotPerBary;
    bt->J_aux[k] = (float)(Gamma_R_prefactor * PLANCK * 1e21 / (4.0 * M_PI) * p->ReionGammaHaloBias / sfr_timescale *
                           p->ReionAlphaUV);
    bt->J_aux_bh[k] = (float)(Gamma_R_prefactor * PLANCK * 1e21 / (4.0 * M_PI) * p->ReionGammaHaloBias /
                              sfr_timescale * p->ReionAlphaUVBH);
    const double G_bh = Gamma_R_prefactor * (SIGMA_HI * p->ReionAlphaUVBH / (p->ReionAlphaUVBH + 2.75) * 1e12);
    Gamma_R_prefactor *= SIGMA_HI * p->ReionAlphaUV / (p->ReionAlphaUV + 2.75) * 1e12;
    bt->G_pref[k] = (float)Gamma_R_prefactor;
    bt->G_pref_bh[k] = (float)G_bh;
    bt->R[k] = (float)R;
    bt->fcoll_pref[k] = p->ReionEfficiency * (4.0 / 3.0) * M_PI / pixel_volume / M_mean * R * R * R;
    // Pop III (find_HII_bubbles.c:443-450): photons per baryon and efficiency of their own
    b3->J_aux[k] = bt->J_aux[k] * (float)(p->ReionNionPhotPerBaryIII / p->ReionNionPhotPerBary);
    b3->G_pref[k] = (float)(Gamma_R_prefactor * p->ReionNionPhotPerBaryIII / p->ReionNionPhotPerBary);
    b3->fcoll_pref[k] = bt->fcoll_pref[k] / p->ReionEfficiency * p->ReionEfficiencyIII;
  }
}

// the grids the z pass tests, in its order (the first ntest of srcs), then in the plain mode
// without recombinations weighted_sfr; returns the count.  weighted_sfr (and effective_bhar) feed
// only Gamma12 on the recombination branch, so without it their filtered fields are never read;
// the plain mode transforms weighted_sfr anyway, as the reference does.
static int hii_sources(const rg_params* p, const rg_grids* g, bool plain, const float** srcs, int* ntest) {
  const bool spin = p->Flag_IncludeSpinTemp != 0, bh = p->Flag_BHFeedback != 0;
  const bool rec = p->Flag_IncludeRecombinations != 0, mini = p->UseMiniHalos != 0;
  int ng = 0;
  srcs[ng++] = g->deltax;
  srcs[ng++] = g->stars;
  if (spin) srcs[ng++] = g->x_e_box;
  if (bh) srcs[ng++] = g->effective_bhm;
  if (mini) srcs[ng++] = g->starsIII;
  if (rec) {
    srcs[ng++] = g->N_rec;
    srcs[ng++] = g->weighted_sfr;
    if (bh) srcs[ng++] = g->effective_bhar;
    if (mini) srcs[ng++] = g->weighted_sfrIII;
  }
  *ntest = ng;
  if (plain && !rec) srcs[ng++] = g->weighted_sfr;
  return ng;
}

static HiiState hii_state(const rg_params* p, const rg_grids* g, uint8_t* state) {
  const bool bh = p->Flag_BHFeedback != 0, mini = p->UseMiniHalos != 0;
  HiiState hs;
  hs.xH = g->xH;
  hs.z_in = g->z_at_ionization;
  hs.J21 = g->J_21_at_ionization;
  hs.temp = g->temp_kinetic_all_gas;
  hs.Tk_box = p->Flag_IncludeSpinTemp ? g->Tk_box : nullptr;
  hs.deltax_unf = g->deltax;
  hs.wsfr = g->weighted_sfr;
  hs.bhar = bh ? g->effective_bhar : nullptr;
  hs.wsfrIII = mini ? g->weighted_sfrIII : nullptr;
  hs.Gamma12 = g->Gamma12;
  hs.r_bubble = g->r_bubble;
  hs.state = state;
  return hs;
}

// the box averages from the reduced sums S (find_HII_bubbles.c:650-700)
static void hii_outputs(const rg_params* p, int nr, const double* S, rg_hii_scalars* out) {
  const bool rec = p->Flag_IncludeRecombinations != 0, mini = p->UseMiniHalos != 0;
  const Units u = make_units(p);
  const double n3 = std::pow((double)p->ReionGridDim, 3);
  const double mass_weight = S[8];
  const double to_msun_yr = p->UnitMass_in_g / u.UnitTime_in_s * SEC_PER_YEAR / SOLAR_MASS;
  out->volume_weighted_global_xH = S[0] / n3;
  out->volume_weighted_global_r_bubble = S[1] / n3;
  out->volume_weighted_global_weighted_sfr = S[2] / n3 * to_msun_yr;
  out->volume_weighted_global_effective_bhar = S[3] / n3 * to_msun_yr;
  out->volume_weighted_global_temp_kinetic_all_gas = S[4] / n3;
  out->mass_weighted_global_xH = S[5] / mass_weight;
  out->mass_weighted_global_r_bubble = S[6] / mass_weight;
  out->mass_weighted_global_temp_kinetic_all_gas = S[7] / mass_weight;
  out->n_radii = nr;
  out->volume_weighted_global_weighted_sfrIII = mini ? S[9] / n3 * to_msun_yr : 0.0;
  const double* R = S + 16;   // recombination sums (find_HII_bubbles.c:666-684)
  out->volume_weighted_global_Gamma12 = rec ? R[2] / n3 : 0.0;
  out->volume_weighted_global_N_rec = rec ? R[4] / n3 : 0.0;
  out->volume_weighted_global_residual_xH = rec ? R[6] / n3 : 0.0;
  out->volume_weighted_global_clumping_factor = rec ? R[8] / n3 : 0.0;
  out->mass_weighted_global_Gamma12 = rec ? R[3] / mass_weight : 0.0;
  out->mass_weighted_global_N_rec = rec ? R[5] / mass_weight : 0.0;
  out->mass_weighted_global_residual_xH = rec ? R[7] / mass_weight : 0.0;
  out->mass_weighted_global_clumping_factor = rec ? R[9] / mass_weight : 0.0;
  if (rec) {
    out->volume_weighted_global_r_bubble = R[0] / n3;
    out->mass_weighted_global_r_bubble = R[1] / mass_weight;
  }
}

// the window table of every radius (and the sharp-k steps) into ctx->wtab / ctx->wcut
static int hii_windows(rg_context* ctx, const rg_params* p, const std::vector<std::pair<double, bool>>& sched,
                       cudaStream_t st) {
  const int N = ctx->N, nr = (int)sched.size();
  const int n2max = 3 * (N / 2) * (N / 2);
  std::vector<double> radii(nr);
  for (int i = 0; i < nr; ++i) radii[i] = sched[i].first;
  int rc;
  if ((rc = ensure_device(ctx, &ctx->d_radii, &ctx->d_radii_elems, (size_t)nr))) return rc;
  RG_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->d_radii, radii.data(), sizeof(double) * nr, cudaMemcpyHostToDevice, st));
  if ((rc = ensure_device(ctx, &ctx->wtab, &ctx->wtab_elems, (size_t)nr * (n2max + 1)))) return rc;
  if ((rc = ensure_device(ctx, &ctx->wcut, &ctx->wcut_elems, (size_t)nr))) return rc;
  return window_table(ctx, p->BoxSize, ctx->d_radii, nr, p->ReionFilterType, ctx->wtab, n2max, st, ctx->wcut);
}

// blocks of the closing pass: enough to fill the chip, at least four cells a thread
static int hii_close_blocks(const rg_context* ctx, int n) {
  return (int)std::max<size_t>(1, std::min((size_t)n * n * n / (4 * CLOSE_NT), (size_t)8 * ctx->num_sms));
}

// radii per batch of the fused mode: the caller's, or 16 where their windowed spectra take at most 6 GB
// and 8 above (fewer launches and less state between batches: 0.34 -> 0.31 ms at 64^3, 4.74 -> 4.53 at
// 192^3, no gain at 512^3), and no more than the device has had room for (hii_buffers)
static int radius_batch(const rg_context* ctx, size_t nc, int ng, int nr) {
  const int kb = ctx->radius_batch > 0 ? ctx->radius_batch : nc * ng * 16 * sizeof(cf) <= ((size_t)6 << 30) ? 16 : 8;
  return std::max(1, std::min({kb, KB_MAX, nr, (int)std::min(ctx->hii_fit / (nc * ng), (size_t)KB_MAX)}));
}

// radii whose window planes are formed at a time: whole batches, at most 256 MB where that is more
// than one
static int plane_radii(int n, int kb, int nr) {
  const int fit = (int)((256u << 20) / (sizeof(float) * wplane_size(n))) / kb * kb;
  return std::min(nr, std::max(kb, fit));
}

// Every buffer of the radius loop over nr radii of nu snapshots (ng grids in all), before the first launch:
// *kb radii a batch, *npl window planes at a time (none for sharp-k).  A batch's spectra and planes grow with
// the batch, so where the device has no room for all of it the two are given back and half the radii are tried:
// the default batch and its planes then need no more than 8 radii without planes did.  A batch that the
// caller set and whose spectra alone do not fit is RG_ENOMEM.  The context remembers what fitted, so that
// later calls do not allocate and free again.
static int hii_buffers(rg_context* ctx, size_t nc, int ng, int nr, int nu, bool planes, size_t npart, int* kb,
                       int* npl) {
  const int N = ctx->N, n2max = 3 * (N / 2) * (N / 2);
  const size_t n3 = (size_t)N * N * N;
  auto all = [&]() -> int {
    int rc = ensure_device(ctx, &ctx->work, &ctx->work_elems, nc * ng * *kb);
    if (!rc) rc = ensure_device(ctx, &ctx->wplanes, &ctx->wplanes_elems, planes ? *npl * wplane_size(N) : 1);
    if (!rc) rc = ensure_device(ctx, &ctx->spec, &ctx->spec_elems, nc * ng);
    // one state byte per cell between radius batches (in words of four)
    if (!rc) rc = ensure_device(ctx, &ctx->bits, &ctx->bits_elems, (n3 * nu + 3) / 4);
    if (!rc) rc = ensure_device(ctx, &ctx->d_radii, &ctx->d_radii_elems, (size_t)nr);
    if (!rc) rc = ensure_device(ctx, &ctx->wtab, &ctx->wtab_elems, (size_t)nr * (n2max + 1));
    if (!rc) rc = ensure_device(ctx, &ctx->wcut, &ctx->wcut_elems, (size_t)nr);
    if (!rc) rc = ensure_device(ctx, &ctx->xy_ctrl, &ctx->xy_ctrl_elems, (size_t)(N / 2 + 1) * *kb + 2);
    if (!rc && !ensure_partials(ctx, npart)) rc = set_error(ctx, RG_ENOMEM, "partials");
    return rc;
  };
  auto release = [](auto** ptr, size_t* elems) {
    if (*ptr) cudaFree(*ptr);
    *ptr = nullptr;
    *elems = 0;
  };
  int rc;
  const size_t fitted = ctx->hii_fit;
  if (ctx->radius_batch > 0 && (rc = ensure_device(ctx, &ctx->work, &ctx->work_elems, nc * ng * *kb))) return rc;
  for (;;) {
    *npl = plane_radii(N, *kb, nr);
    rc = all();
    if (rc == RG_ENOMEM && planes && *npl > *kb) {
      *npl = *kb;
      rc = all();
    }
    if (rc == RG_ENOMEM && *kb == 1) ctx->hii_fit = fitted;   // nothing fitted: a later call tries anew
    if (rc != RG_ENOMEM || *kb == 1) return rc;
    release(&ctx->work, &ctx->work_elems);
    release(&ctx->wplanes, &ctx->wplanes_elems);
    *kb /= 2;
    ctx->hii_fit = nc * ng * *kb;
  }
}

int hii_snapshot(rg_context* ctx, const rg_params* p, const rg_snapshot* s, const rg_grids* g, rg_hii_scalars* out,
                 const Staging* stg) {
  const Staging none;
  if (!stg) stg = &none;
  int rc;
  cudaStream_t st = ctx->stream;
  const int N = ctx->N;
  const bool rec = p->Flag_IncludeRecombinations != 0;
  const double redshift = s->ZZ[s->snapshot];
  HiiConst c;
  if ((rc = hii_const(ctx, p, redshift, &c))) return rc;

  const float* srcs[10];
  int ntest = 0;
  const bool plain = ctx->mode == RG_MODE_PLAIN;
  const int ng = hii_sources(p, g, plain, srcs, &ntest);

  const size_t nc = (size_t)(N / 2 + 1) * N * N;
  auto sched = radius_schedule(p, redshift);
  const int nr = (int)sched.size();
  int kb = plain ? 1 : radius_batch(ctx, nc, ng, nr);
  const int cb = hii_close_blocks(ctx, N);
  int npl = 0;
  if ((rc = hii_buffers(ctx, nc, ng, nr, 1, p->ReionFilterType != 1,
                        std::max((size_t)cb * HII_NSUM, (size_t)4 * ctx->num_sms * REC_NSUM), &kb, &npl)))
    return rc;
  double* partials = ctx->partials;
  if ((rc = stage_wait(ctx, stg->inputs, st))) return rc;
  const int fg = fft_forward_group(N);   // grids per forward launch
  for (int g0 = 0; g0 < ng; g0 += fg)
    if ((rc = fft_forward(ctx, N, srcs + g0, std::min(fg, ng - g0), ctx->spec + nc * g0, nc,
                          1.0 / std::pow((double)N, 3), st)))
      return rc;

  if ((rc = hii_windows(ctx, p, sched, st))) return rc;
  const int n2max = 3 * (N / 2) * (N / 2);
  const int* wcut = p->ReionFilterType == 1 ? ctx->wcut : nullptr;

  // r_bubble is only written on the recombination branch: zero it once
  RG_CUDA_TRY(ctx, cudaMemsetAsync(g->r_bubble, 0, sizeof(float) * (size_t)N * N * N, st));
  if (stg->host_r_bubble && !rec) {
    // final already: the host copy overlaps the radius loop
    cudaEvent_t e;
    if ((rc = stage_record(ctx, 4, st, &e))) return rc;
    RG_CUDA_TRY(ctx, cudaStreamWaitEvent(ctx->copy_stream, e, 0));
    RG_CUDA_TRY(ctx, cudaMemcpyAsync(stg->host_r_bubble, g->r_bubble, sizeof(float) * (size_t)N * N * N,
                                     cudaMemcpyDeviceToHost, ctx->copy_stream));
  }
  const HiiState hs = hii_state(p, g, reinterpret_cast<uint8_t*>(ctx->bits));

  if ((rc = xy_ctrl_reset(ctx, (size_t)(N / 2 + 1) * kb, st))) return rc;
  for (int r0 = 0; r0 < nr; r0 += kb) {
    const int cnt = std::min(kb, nr - r0);
    const bool fin = (r0 + cnt == nr);
    HiiZUnits us;
    HiiBatchIII b3;
    hii_batch_radii(p, redshift, sched, r0, cnt, ntest, &us.u[0].bt, &b3);
    us.u[0].c = c;
    us.u[0].s = hs;
    // the snapshot's last radius is unfiltered (find_HII_bubbles.c:313)
    const int unf = fin ? cnt - 1 : -1;
    if (!wcut && r0 % npl == 0 &&
        (rc = window_planes(ctx, N, ctx->wtab + (size_t)r0 * (n2max + 1), std::min(npl, nr - r0), ctx->wplanes, st)))
      return rc;
    if ((rc = inverse_xy(ctx, N, ctx->spec, ng, ng, ctx->work, nc, cnt, ctx->wplanes + (r0 % npl) * wplane_size(N),
                         unf, st, wcut ? wcut + r0 : nullptr)))
      return rc;
    if (r0 == 0 && (rc = stage_wait(ctx, stg->state, st))) return rc;
    if ((rc = hii_z(ctx, N, ctx->work, nc, ntest, 1, us, b3, st))) return rc;
  }
  if ((rc = stage_wait(ctx, stg->closing, st))) return rc;
  if ((rc = hii_close(ctx, N, &c, &hs, 1, partials, cb, st))) return rc;
  if ((rc = reduce_partials(ctx, partials, cb, HII_NSUM, ctx->d_sums, st))) return rc;
  if (rec) {
    RecTables tab;
    tab.knots = ctx->rec_knots;
    tab.y = ctx->rec_y;
    tab.c = ctx->rec_c;
    tab.nz = ctx->rec_nz;
    tab.nt = ctx->rec_nt;
    tab.ng = ctx->rec_ng;
    // recombinations.c:51-64: the table's bounds as the float expressions of the C
    tab.lng_lo = (double)(-10.0f);
    tab.lng_hi = (double)(-10.0f + 0.1f * (float)(ctx->rec_ng - 1));
    RecConst rcst;
    rcst.redshift = redshift;
    rcst.hubble_h = p->Hubble_h;
    const double prev_z = s->snapshot == 0 ? redshift : s->ZZ[s->snapshot - 1];
    rcst.zstep = (float)(prev_z - redshift);
    rcst.fabs_dtdz = (float)std::fabs(dtdz(p, (float)redshift) / p->Hubble_h);
    rcst.temp_dep = p->Flag_TemperatureDependentRec != 0;
    RecState rs;
    rs.xH = g->xH;
    rs.temp = g->temp_kinetic_all_gas;
    rs.deltax_unf = g->deltax;
    rs.r_bubble = g->r_bubble;
    rs.Gamma12 = g->Gamma12;
    rs.N_rec = g->N_rec;
    rs.residual_xH = g->residual_xH;
    rs.clumping_factor = g->clumping_factor;
    rs.t_resp = g->t_resp;
    const int rb = 4 * ctx->num_sms;
    if ((rc = hii_recomb(ctx, N, tab, rcst, rs, partials, rb, st))) return rc;
    if ((rc = reduce_partials(ctx, partials, rb, REC_NSUM, ctx->d_sums + 16, st))) return rc;
  }
  RG_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_sums, ctx->d_sums, sizeof(double) * 32, cudaMemcpyDeviceToHost, st));
  if ((rc = xy_ctrl_fetch(ctx, st))) return rc;
  RG_CUDA_TRY(ctx, cudaStreamSynchronize(st));
  prof_resolve(ctx);
  if ((rc = xy_ctrl_result(ctx))) return rc;
  hii_outputs(p, nr, ctx->h_sums, out);
  return RG_OK;
}

int hii_batch(rg_context* ctx, int nu, const rg_params* p, const rg_snapshot* s, const rg_grids* g,
              rg_hii_scalars* out) {
  int rc;
  cudaStream_t st = ctx->stream;
  const int N = ctx->N;
  const double z0 = s[0].ZZ[s[0].snapshot];
  auto sched = radius_schedule(&p[0], z0);
  for (int u = 1; u < nu; ++u) {
    auto su = radius_schedule(&p[u], s[u].ZZ[s[u].snapshot]);
    if (su.size() != sched.size()) return set_error(ctx, RG_EINVAL, "batch units with different radius schedules");
    for (size_t i = 0; i < su.size(); ++i)
      if (su[i].first != sched[i].first) return set_error(ctx, RG_EINVAL, "batch units with different radii");
  }
  std::vector<HiiConst> cs(nu);
  for (int u = 0; u < nu; ++u)
    if ((rc = hii_const(ctx, &p[u], s[u].ZZ[s[u].snapshot], &cs[u]))) return rc;
  // the units' grids one after another: unit u's grid k is grid u ngu + k of the batch
  const float* one[10];
  int ntest = 0;
  const int ngu = hii_sources(&p[0], &g[0], false, one, &ntest);
  std::vector<const float*> srcs((size_t)nu * ngu);
  for (int u = 0; u < nu; ++u) {
    hii_sources(&p[u], &g[u], false, one, &ntest);
    for (int k = 0; k < ngu; ++k) srcs[(size_t)u * ngu + k] = one[k];
  }
  const int ng = nu * ngu;
  const size_t nc = (size_t)(N / 2 + 1) * N * N, n3 = (size_t)N * N * N;
  const int nr = (int)sched.size();
  int kb = radius_batch(ctx, nc, ng, nr);
  const int cb = hii_close_blocks(ctx, N);
  int npl = 0;
  if ((rc = hii_buffers(ctx, nc, ng, nr, nu, p[0].ReionFilterType != 1, (size_t)nu * cb * HII_NSUM, &kb, &npl)))
    return rc;
  double* partials = ctx->partials;
  if ((rc = ensure_device(ctx, &ctx->batch_sums, &ctx->batch_sums_elems, (size_t)32 * nu))) return rc;
  if ((size_t)nu > ctx->h_batch_sums_elems) {
    if (ctx->h_batch_sums) cudaFreeHost(ctx->h_batch_sums);
    ctx->h_batch_sums = nullptr;
    ctx->h_batch_sums_elems = 0;
    if (cudaMallocHost((void**)&ctx->h_batch_sums, sizeof(double) * 32 * nu) != cudaSuccess)
      return set_error(ctx, RG_ENOMEM, "pinned batch sums");
    ctx->h_batch_sums_elems = (size_t)nu;
  }
  const int fg = fft_forward_group(N);
  for (int g0 = 0; g0 < ng; g0 += fg)
    if ((rc = fft_forward(ctx, N, srcs.data() + g0, std::min(fg, ng - g0), ctx->spec + nc * g0, nc,
                          1.0 / std::pow((double)N, 3), st)))
      return rc;
  if ((rc = hii_windows(ctx, &p[0], sched, st))) return rc;
  const int n2max = 3 * (N / 2) * (N / 2);
  const int* wcut = p[0].ReionFilterType == 1 ? ctx->wcut : nullptr;
  for (int u = 0; u < nu; ++u)
    RG_CUDA_TRY(ctx, cudaMemsetAsync(g[u].r_bubble, 0, sizeof(float) * n3, st));
  std::vector<HiiState> hs(nu);
  for (int u = 0; u < nu; ++u)
    hs[u] = hii_state(&p[u], &g[u], reinterpret_cast<uint8_t*>(ctx->bits) + n3 * u);

  if ((rc = xy_ctrl_reset(ctx, (size_t)(N / 2 + 1) * kb, st))) return rc;
  const int zu = hii_z_units(N);
  for (int r0 = 0; r0 < nr; r0 += kb) {
    const int cnt = std::min(kb, nr - r0);
    const bool fin = (r0 + cnt == nr);
    const int unf = fin ? cnt - 1 : -1;
    // the windowed inverse x/y passes of every unit's grids in one launch; unit u's block of
    // the work buffer is [radius][its grids], as a single snapshot's
    if (!wcut && r0 % npl == 0 &&
        (rc = window_planes(ctx, N, ctx->wtab + (size_t)r0 * (n2max + 1), std::min(npl, nr - r0), ctx->wplanes, st)))
      return rc;
    if ((rc = inverse_xy(ctx, N, ctx->spec, ng, ngu, ctx->work, nc, cnt, ctx->wplanes + (r0 % npl) * wplane_size(N),
                         unf, st, wcut ? wcut + r0 : nullptr)))
      return rc;
    // the z passes, zu snapshots a launch (a 96^3 box alone fills a fifth of the chip)
    for (int u0 = 0; u0 < nu; u0 += zu) {
      const int cu = std::min(zu, nu - u0);
      HiiZUnits us;
      HiiBatchIII b3;
      for (int k = 0; k < cu; ++k) {
        const int u = u0 + k;
        hii_batch_radii(&p[u], s[u].ZZ[s[u].snapshot], sched, r0, cnt, ntest, &us.u[k].bt, &b3);
        us.u[k].c = cs[u];
        us.u[k].s = hs[u];
      }
      if ((rc = hii_z(ctx, N, ctx->work + (size_t)u0 * cnt * ngu * nc, nc, ntest, cu, us, b3, st)))
        return rc;
    }
  }
  if ((rc = hii_close(ctx, N, cs.data(), hs.data(), nu, partials, cb, st))) return rc;
  if ((rc = reduce_partials(ctx, partials, cb, HII_NSUM, ctx->batch_sums, st, nu, (size_t)cb * HII_NSUM, 32))) return rc;
  RG_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_batch_sums, ctx->batch_sums, sizeof(double) * 32 * nu,
                                   cudaMemcpyDeviceToHost, st));
  if ((rc = xy_ctrl_fetch(ctx, st))) return rc;
  RG_CUDA_TRY(ctx, cudaStreamSynchronize(st));
  prof_resolve(ctx);
  if ((rc = xy_ctrl_result(ctx))) return rc;
  for (int u = 0; u < nu; ++u) hii_outputs(&p[u], nr, ctx->h_batch_sums + 32 * u, &out[u]);
  return RG_OK;
}

static int debug_inverse(rg_context* ctx, int n, const float* wplane, float* d_out, cudaStream_t st) {
  RG_DISPATCH_N(n, launch_debug_inverse<NN>(ctx, ctx->spec, ctx->work, wplane, d_out, st));
}

int spectrum_to_padded(rg_context* ctx, float* d_out, cudaStream_t st) {
  const size_t nc = (size_t)(ctx->N / 2 + 1) * ctx->N * ctx->N;
  int rc;
  if ((rc = ensure_device(ctx, &ctx->work, &ctx->work_elems, nc))) return rc;
  return debug_inverse(ctx, ctx->N, nullptr, d_out, st);
}

int debug_roundtrip(rg_context* ctx, const rg_params* p, const float* d_in, float* d_out, double R, int ftype) {
  int rc;
  cudaStream_t st = ctx->stream;
  const int N = ctx->N;
  const size_t nc = (size_t)(N / 2 + 1) * N * N;
  if ((rc = ensure_device(ctx, &ctx->spec, &ctx->spec_elems, nc))) return rc;
  if ((rc = ensure_device(ctx, &ctx->work, &ctx->work_elems, nc))) return rc;
  const float* srcs[1] = {d_in};
  if ((rc = fft_forward(ctx, N, srcs, 1, ctx->spec, nc, 1.0 / std::pow((double)N, 3), st))) return rc;
  const float* wplane = nullptr;
  if (ftype >= 0) {
    if ((rc = ensure_device(ctx, &ctx->wplanes, &ctx->wplanes_elems, wplane_size(N)))) return rc;
    prof_begin(ctx, "window_planes", st);
    k_window_plane<<<dim3(N / 2 + 1, N / 2 + 1), 64, 0, st>>>(2.0 * M_PI / p->BoxSize, R, ftype, N, ctx->wplanes);
    prof_end(ctx, 4.0 * wplane_size(N), st);
    RG_CUDA_TRY(ctx, cudaGetLastError());
    wplane = ctx->wplanes;
  }
  if ((rc = debug_inverse(ctx, N, wplane, d_out, st))) return rc;
  return xy_ctrl_check(ctx, st);
}

}  // namespace rg
