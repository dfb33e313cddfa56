// 21-cm brightness temperature, ComputeBrightnessTemperatureBox()
// (src/core/BrightnessTemperature.c:24-124,512-548) without peculiar velocities: one pass
// over the cells, with the FP64 volume average reduced in the same kernel.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "rg_internal.h"
#include "rg_pass.cuh"
#include "rg_xray.h"

namespace rg {

constexpr int DT_NT = 256;
constexpr int N_RSD_STEPS = 50;      // reionization.h:34
constexpr float MAX_DVDR = 0.2f;     // reionization.h:45

// FP64 block sum in a fixed order -> partials[blockIdx.x]
__device__ __forceinline__ void dt_block_sum(double acc, double* __restrict__ partials) {
  __shared__ double sh[DT_NT / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if (threadIdx.x % 32 == 0) sh[threadIdx.x / 32] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double v = 0.0;
#pragma unroll
    for (int w = 0; w < DT_NT / 32; ++w) v += sh[w];
    partials[blockIdx.x] = v;
  }
}

// f(cell, padded cell) over the box, DT_U cells of a thread in a row of the loop so that their loads are
// in flight together (one at a time a pass over 256^3 cells reached 2.5 of 6.5 TB/s)
constexpr int DT_U = 4;
__device__ __forceinline__ size_t dt_padded(size_t ir, int n) {
  return ir + ((unsigned)ir / (unsigned)n) * 2;   // rows of n + 2 values (n is even, at most 512)
}

__global__ void __launch_bounds__(DT_NT) k_delta_T(const float* __restrict__ xH, const float* __restrict__ deltax,
                                                   const float* __restrict__ TS, float* __restrict__ dT, int n,
                                                   float const_factor, double t_rad, int spin, int pec_vel_gt1,
                                                   float redshift, double* __restrict__ partials) {
  const size_t n3 = (size_t)n * n * n, step = (size_t)gridDim.x * DT_NT;
  const double opz = 1. + (double)redshift;
  double acc = 0.0;
  for (size_t i0 = (size_t)blockIdx.x * DT_NT + threadIdx.x; i0 < n3; i0 += DT_U * step) {
    float x[DT_U], d[DT_U], t[DT_U];
#pragma unroll
    for (int k = 0; k < DT_U; ++k) {
      const size_t i = i0 + k * step;
      if (i >= n3) break;
      x[k] = xH[i];
      d[k] = deltax[dt_padded(i, n)];
      t[k] = spin ? TS[i] : 1.f;
    }
#pragma unroll
    for (int k = 0; k < DT_U; ++k) {
      const size_t i = i0 + k * step;
      if (i >= n3) break;
      float v = (float)((double)const_factor * (double)x[k] * (1.0 + (double)d[k]));
      if (spin) {
        if (pec_vel_gt1) {
          v = (float)((double)v * (opz / (1000. * (double)t[k])));
        } else {
          const double fac = 1 - t_rad / (double)t[k];
          v = (float)((double)v * fac);
        }
      }
      dT[i] = v;
      acc += (double)v;
    }
  }
  dt_block_sum(acc, partials);
}

int delta_T_launch(rg_context* ctx, int n, const float* xH, const float* deltax, const float* TS, float* dT,
                   float const_factor, double t_rad, int spin, int pec_gt1, float redshift, double* partials,
                   int nblocks, cudaStream_t st) {
  prof_begin(ctx, "delta_T", st);
  k_delta_T<<<nblocks, DT_NT, 0, st>>>(xH, deltax, TS, dT, n, const_factor, t_rad, spin, pec_gt1, redshift, partials);
  // xH, deltax (and TS) read, delta_T written
  prof_end(ctx, (double)n * n * n * (spin ? 16.0 : 12.0), st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  return RG_OK;
}

// ---------------------------------------------------------------------------
// peculiar velocities (BrightnessTemperature.c:150-509): with the spin temperature,
// Flag_IncludePecVelsFor21cm 1 caps the velocity gradient (the 21cmFAST treatment), 2 uses the
// optical-depth form with the uncapped gradient, 3 adds the line-of-sight re-binning of 50
// sub-cells per cell (Greig & Mesinger 2018).  The values are floats where the reference's are, and each
// step is taken in double as there, with products by reciprocals in place of its divisions by constants
// (an ulp of double) and the re-binning in closed form (k_rsd).

// velocity in the tree code's units -> comoving velocity (BrightnessTemperature.c:173-196); the
// padding of each row is not touched (the r2c transform ignores it).  f0 is the factor of the tree
// code's units, f1 that of cm in Mpc, and the division by 1 / (1 + z) a product with 1 + z.
__global__ void __launch_bounds__(DT_NT) k_vel_convert(const float* __restrict__ vel, float* __restrict__ vc, int n,
                                                       int trees, double f0, double f1, double opz) {
  const size_t n3 = (size_t)n * n * n, step = (size_t)gridDim.x * DT_NT;
  for (size_t i0 = (size_t)blockIdx.x * DT_NT + threadIdx.x; i0 < n3; i0 += DT_U * step) {
    float in[DT_U];
#pragma unroll
    for (int k = 0; k < DT_U; ++k) {
      const size_t i = i0 + k * step;
      if (i >= n3) break;
      in[k] = vel[dt_padded(i, n)];
    }
#pragma unroll
    for (int k = 0; k < DT_U; ++k) {
      const size_t i = i0 + k * step;
      if (i >= n3) break;
      float v = in[k];
      if (trees == 1) v = (float)(f0 * (double)v / 1000.);
      else v = (float)(f0 * (double)v);
      v = (float)((double)v * f1);
      vc[dt_padded(i, n)] = (float)((double)v * opz);
    }
  }
}

// the spectrum of the velocity: / N^3, * Hubble_h (BrightnessTemperature.c:206-213), then * i k_z
// (velocity_gradient, reionization.c:3435-3450); S[kz][x][y]
__global__ void __launch_bounds__(DT_NT) k_vel_grad_spec(cf* __restrict__ spec, int n, double n3, double h, float dk) {
  const size_t total = (size_t)(n / 2 + 1) * n * n;
  for (size_t i = (size_t)blockIdx.x * DT_NT + threadIdx.x; i < total; i += (size_t)gridDim.x * DT_NT) {
    const int kz = (int)(i / ((size_t)n * n));
    const cf v = spec[i];
    float re = (float)((double)v.x / n3), im = (float)((double)v.y / n3);
    re = (float)((double)re * h);
    im = (float)((double)im * h);
    const float k = (float)kz * dk;
    // (re + i im) (0 + i k)
    spec[i] = cf{__fsub_rn(__fmul_rn(re, 0.f), __fmul_rn(im, k)), __fadd_rn(__fmul_rn(re, k), __fmul_rn(im, 0.f))};
  }
}

// the gradient correction of delta_T (BrightnessTemperature.c:215-305, spin temperature on), with the
// FP64 sum of the result
__global__ void __launch_bounds__(DT_NT) k_vel_correct(float* __restrict__ dT, const float* __restrict__ grad,
                                                       const float* __restrict__ TS, int n, int flag, float H_z,
                                                       double t_rad, float redshift, double* __restrict__ partials) {
  const size_t n3 = (size_t)n * n * n, step = (size_t)gridDim.x * DT_NT;
  const double max_v_deriv = fabs((double)(MAX_DVDR * H_z));
  const double inv_H = 1.0 / (double)H_z, f = 1000. / (1. + (double)redshift);
  double acc = 0.0;
  for (size_t i0 = (size_t)blockIdx.x * DT_NT + threadIdx.x; i0 < n3; i0 += DT_U * step) {
    float d[DT_U], gr[DT_U], t[DT_U];
#pragma unroll
    for (int k = 0; k < DT_U; ++k) {
      const size_t i = i0 + k * step;
      if (i >= n3) break;
      d[k] = dT[i];
      gr[k] = grad[dt_padded(i, n)];
      t[k] = flag == 1 ? 0.f : TS[i];
    }
#pragma unroll
    for (int k = 0; k < DT_U; ++k) {
      const size_t i = i0 + k * step;
      if (i >= n3) break;
      const double g = (double)gr[k];
      float v;
      if (flag == 1) {
        double dvdx = g;
        if (fabs(dvdx) > max_v_deriv) dvdx = dvdx < 0 ? -max_v_deriv : max_v_deriv;
        v = (float)((double)d[k] / (dvdx * inv_H + 1.0));
      } else {
        const double gc = fabs(g * inv_H + 1.0);
        const double ts = ((double)t[k] - t_rad) * f;
        v = gc < FRACT_FLOAT_ERR ? (float)ts : (float)((1. - exp(-(double)d[k] / gc)) * ts);
      }
      dT[i] = v;
      acc += (double)v;
    }
  }
  dt_block_sum(acc, partials);
}

struct RsdConst {
  float x_pos[N_RSD_STEPS];          // sub-cell centres in cell widths
  float x_pos_offset[N_RSD_STEPS];   // ... in Mpc
  double inv_cell;                   // 1 / cell width, Mpc^-1
  double inv_w_sub, half;            // sub-cell width (inverse) and half width in cell widths
  float H_z;
  int n_low;                         // sub-cells up to the cell's centre
};

// line-of-sight re-binning (BrightnessTemperature.c:307-509): every contributing cell moves its 50
// sub-cells by the interpolated displacement v / H(z) and adds each (or its two parts) to the cells it
// lands in, periodically along z.  A block takes whole (x, y) lines, whose sums live in shared memory;
// the adds of different cells meet there in any order.
//
// The displacement is linear between cell centres, so on either side of a cell's centre the sub-cells
// (length 1 in units of their width) start at L_s = U + s g, g = 1 + the change of the displacement
// over a cell.  What of them lies left of a boundary B is
//   F(B) = sum_s clamp(B - L_s, 0, 1) = n1 + sum over n1 <= s < n2 of (B - U - s g),
// n1 sub-cells wholly left of B and n2 that reach it: a closed form in FP64, and a cell gets F(right
// edge) - F(left edge).  Two or three cells a side instead of 50 sub-cells with one or two shared-memory
// adds each (compare-and-swap loops, in divergent branches): 3.17 -> 0.51 ms at 256^3; on velocities that
// cross and spread the sub-cells everywhere (white noise, 512^3) 43.0 -> 6.4 ms, and 51.2 with those cells one
// by one.  Where they spread over more than 16 cells a side (|g| beyond 32) or are far off, infinite or not
// numbers, they are moved one by one as in the reference.
__global__ void __launch_bounds__(DT_NT) k_rsd(float* __restrict__ dT, const float* __restrict__ xH,
                                               const float* __restrict__ vc, int n, int lines, const RsdConst c,
                                               double* __restrict__ partials) {
  extern __shared__ float acc[];
  constexpr double NS = N_RSD_STEPS;
  const int padw = n + 2;
  const size_t nrows = (size_t)n * n;
  auto wrap = [n](int k) { return ((k % n) + n) % n; };   // the reference's periodic index
  double total = 0.0;
  for (size_t row0 = (size_t)blockIdx.x * lines; row0 < nrows; row0 += (size_t)gridDim.x * lines) {
    const int cells = (int)min((size_t)lines, nrows - row0) * n;
    for (int i = threadIdx.x; i < cells; i += DT_NT) acc[i] = 0.f;
    __syncthreads();
    for (int i = threadIdx.x; i < cells; i += DT_NT) {
      const int ln = i / n, kk = i - ln * n;
      const size_t row = row0 + ln;
      float* line = acc + ln * n;
      const float* v = vc + row * padw;
      const float d = dT[row * n + kk];
      if (!(fabs((double)d) >= FRACT_FLOAT_ERR && (double)xH[row * n + kk] >= FRACT_FLOAT_ERR)) continue;
      // displacements at the previous cell's, this and the next cell's centre, Mpc
      const double d1 = (double)(v[kk == 0 ? n - 1 : kk - 1] / c.H_z);
      const double d2 = (double)(v[kk] / c.H_z);
      const double d3 = (double)(v[kk == n - 1 ? 0 : kk + 1] / c.H_z);
      const double dd = (double)d / NS;
      const double slope[2] = {(d2 - d1) * c.inv_cell, (d3 - d2) * c.inv_cell};
      const double U[2] = {NS * d1 * c.inv_cell + 0.5 * NS * slope[0] + 0.5 * (1.0 + slope[0]) - 0.5,
                           NS * d2 * c.inv_cell - 0.5 * NS * slope[1] + (c.n_low + 0.5) * (1.0 + slope[1]) - 0.5};
      const double g0 = 1.0 + slope[0], g1 = 1.0 + slope[1];
      if (fabs(g0) <= 32.0 && fabs(g1) <= 32.0 && fabs(U[0]) < 5e10 && fabs(U[1]) < 5e10) {
        int cur = 0;   // the cell, relative to kk, whose share is kept
        double share = 0.0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int m = h ? N_RSD_STEPS - c.n_low : c.n_low;
          // crossed sub-cells (g < 0) counted from their other end; g = 0: the infinities and NaN of
          // inv_g end at the bounds of n1 and n2
          const double gs = h ? g1 : g0, g = fabs(gs), inv_g = 1.0 / g, L0 = gs < 0.0 ? U[h] + (m - 1) * gs : U[h];
          const int k0 = (int)floor(L0 * (1.0 / NS)), k1 = (int)floor((L0 + (m - 1) * g + 1.0) * (1.0 / NS));
          double left = 0.0;
          for (int k = k0; k <= k1; ++k) {
            double f = m;
            if (k < k1) {
              const double t = NS * (k + 1.0) - L0;
              const double n1 = fmin(fmax(floor((t - 1.0) * inv_g) + 1.0, 0.0), (double)m);
              const double n2 = fmin(fmax(ceil(t * inv_g), n1), (double)m);
              f = n1 + (n2 - n1) * t - 0.5 * g * (n2 * (n2 - 1.0) - n1 * (n1 - 1.0));
            }
            if (k != cur) {
              if (share != 0.0) atomicAdd(line + wrap(kk + cur), (float)(share * dd));
              cur = k;
              share = 0.0;
            }
            share += f - left;
            left = f;
          }
        }
        if (share != 0.0) atomicAdd(line + wrap(kk + cur), (float)(share * dd));
        continue;
      }
      const float val = d / (float)N_RSD_STEPS;
      auto put = [&](int k, double frac) { atomicAdd(line + wrap(k), (float)(frac * dd)); };
      for (int s = 0; s < N_RSD_STEPS; ++s) {
        const double xp = (double)c.x_pos[s];
        const double disp = s < c.n_low ? d1 + (xp + 0.5) * (d2 - d1) : d2 + (xp - 0.5) * (d3 - d2);
        const double pos = ((double)c.x_pos_offset[s] + disp) * c.inv_cell;
        const double lo = pos - c.half, hi = pos + c.half;
        if (lo >= 0.0 && hi < 1.0) {
          atomicAdd(line + kk, val);
        } else if (lo < 0.0 && hi < 0.0) {
          const double cd = ceil(fabs(lo)) - 1.;
          const int ic = (int)cd;
          if (fabs(hi) > cd) {
            atomicAdd(line + wrap(kk - (ic + 1)), val);
          } else {
            const double fo = (fabs(lo) - cd) * c.inv_w_sub;
            put(kk - ic, 1. - fo);
            put(kk - (ic + 1), fo);
          }
        } else if (lo < 0.0 && (hi > 0.0 && hi < 1.0)) {
          const double fw = hi * c.inv_w_sub;
          put(kk - 1, 1. - fw);
          put(kk, fw);
        } else {
          const double cd = floor(fabs(hi));
          const int ic = (int)cd;
          if (lo >= cd) {
            atomicAdd(line + wrap(kk + ic), val);
          } else {
            const double fo = (hi - cd) * c.inv_w_sub;
            put(kk + ic - 1, 1. - fo);
            put(kk + ic, fo);
          }
        }
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < cells; i += DT_NT) {
      const float v = acc[i];
      dT[row0 * n + i] = v;
      total += (double)v;
    }
    __syncthreads();   // the lines are read before the next ones are zeroed
  }
  dt_block_sum(total, partials);
}

// the velocity stages after k_delta_T; leaves the FP64 sum of the final delta_T in partials
static int velocity_modes(rg_context* ctx, const rg_params* p, const rg_grids* g, float redshift, double t_rad,
                          int nblocks, cudaStream_t st) {
  const int n = ctx->N;
  const int flag = p->Flag_IncludePecVelsFor21cm;
  const size_t nc = (size_t)(n / 2 + 1) * n * n, npad = 2 * nc, n3 = (size_t)n * n * n;
  int rc;
  if ((rc = ensure_device(ctx, &ctx->vel_work, &ctx->vel_work_elems, 2 * npad))) return rc;
  if ((rc = ensure_device(ctx, &ctx->spec, &ctx->spec_elems, nc))) return rc;
  float* vc = ctx->vel_work;
  float* grad = ctx->vel_work + npad;
  const Cosmo cm(p);
  const float H_z = (float)cm.hubble(redshift);
  prof_begin(ctx, "vel_convert", st);
  const double opz = 1. + (double)redshift;
  k_vel_convert<<<nblocks, DT_NT, 0, st>>>(g->vel, vc, n, p->TreesID, p->TreesID == 1 ? std::sqrt(1. / opz) : opz,
                                           1000. * 100. / MPC, opz);
  prof_end(ctx, 8.0 * n3, st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  const float* src = vc;
  if ((rc = fft_forward(ctx, n, &src, 1, ctx->spec, nc, 1.0, st))) return rc;
  const float dk = (float)(2.0 * M_PI / (float)p->BoxSize);
  prof_begin(ctx, "vel_gradient", st);
  k_vel_grad_spec<<<nblocks, DT_NT, 0, st>>>(ctx->spec, n, std::pow((double)n, 3), p->Hubble_h, dk);
  prof_end(ctx, 16.0 * nc, st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  if ((rc = xy_ctrl_reset(ctx, (size_t)(n / 2 + 1), st))) return rc;
  if ((rc = spectrum_to_padded(ctx, grad, st))) return rc;
  prof_begin(ctx, "vel_correct", st);
  k_vel_correct<<<nblocks, DT_NT, 0, st>>>(g->delta_T, grad, g->TS_box, n, flag, H_z, t_rad, redshift,
                                           ctx->partials);
  prof_end(ctx, 16.0 * n3, st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  if (flag == 3) {
    RsdConst c;
    const double box = p->BoxSize / p->Hubble_h;   // Mpc
    const double sub_w = (box / ((double)n)) / (double)N_RSD_STEPS;
    const double cell = box / (float)n;
    c.inv_cell = 1.0 / cell;
    c.inv_w_sub = cell / sub_w;
    c.half = (sub_w / 2.) / cell;
    c.H_z = H_z;
    c.n_low = 0;
    for (int i = 0; i < N_RSD_STEPS; ++i) {
      c.x_pos_offset[i] = (float)(sub_w * (float)i + sub_w / 2.);
      c.x_pos[i] = (float)(c.x_pos_offset[i] / (box / (float)n));
      // up to 0.5 between the previous cell's centre and this one's, beyond between this and the next
      if ((double)c.x_pos[i] <= 0.5) c.n_low = i + 1;
    }
    // whole lines a block: 256 cells or one line
    const int lines = std::max(1, DT_NT / n);
    prof_begin(ctx, "rsd_los", st);
    k_rsd<<<nblocks, DT_NT, sizeof(float) * n * lines, st>>>(g->delta_T, g->xH, vc, n, lines, c, ctx->partials);
    prof_end(ctx, 16.0 * n3, st);
    RG_CUDA_TRY(ctx, cudaGetLastError());
  }
  return RG_OK;
}

}  // namespace rg

using namespace rg;


extern "C" {

int rg_delta_T(rg_context* ctx, const rg_params* p, const rg_snapshot* s, const rg_grids* g, double* volume_ave_Tb) {
  if (!ctx || !p || !s || !g || !volume_ave_Tb || !s->ZZ) return RG_EINVAL;
  if (p->ReionGridDim != ctx->N) return set_error(ctx, RG_EINVAL, "ReionGridDim differs from the context's grid");
  if (s->snapshot < 0 || s->snapshot >= s->n_snapshots) return set_error(ctx, RG_EINVAL, "snapshot out of range");
  if (p->Flag_IncludePecVelsFor21cm < 0 || p->Flag_IncludePecVelsFor21cm > 3)
    return set_error(ctx, RG_EINVAL, "Flag_IncludePecVelsFor21cm must be 0, 1, 2 or 3");
  if (p->UseMiniHalos)
    return set_error(ctx, RG_EUNSUPPORTED, "UseMiniHalos: the Pop II brightness temperature delta_TII is not built");
  const bool vel_modes = p->Flag_IncludeSpinTemp && p->Flag_IncludePecVelsFor21cm > 0;
  if (!g->xH || !g->deltax || !g->delta_T || (p->Flag_IncludeSpinTemp && !g->TS_box) || (vel_modes && !g->vel))
    return set_error(ctx, RG_EINVAL, "missing grid pointer");
  if (vel_modes && (p->TreesID < 0 || p->TreesID > 2)) return set_error(ctx, RG_EINVAL, "TreesID must be 0, 1 or 2");
  if (vel_modes && !(p->Hubble_h > 0)) return set_error(ctx, RG_EINVAL, "Hubble_h must be positive");
  cudaSetDevice(ctx->device);
  cudaStream_t st = ctx->stream;
  const int n = ctx->N;
  // BrightnessTemperature.c:49-54, 82: float parameters, double expression
  const float redshift = (float)s->ZZ[s->snapshot];
  const float Hubble_h = (float)p->Hubble_h;
  const float OmegaM = (float)p->OmegaM;
  const float OmegaB = (float)(OmegaM * p->BaryonFrac);
  const float const_factor = (float)(27.0 * ((double)(OmegaB * Hubble_h * Hubble_h) / 0.023) *
                                     std::sqrt((0.15 / (double)OmegaM / (double)Hubble_h / (double)Hubble_h) *
                                               (1.0 + (double)redshift) / 10.0));
  const double t_rad = TCMB * (1. + (double)redshift);
  const int nblocks = 148 * 8;
  if (!ensure_partials(ctx, (size_t)nblocks)) return set_error(ctx, RG_ENOMEM, "partials");
  int rc = delta_T_launch(ctx, n, g->xH, g->deltax, g->TS_box, g->delta_T, const_factor, t_rad,
                          p->Flag_IncludeSpinTemp, p->Flag_IncludePecVelsFor21cm > 1, redshift, ctx->partials,
                          nblocks, st);
  if (rc) return rc;
  if (vel_modes && (rc = velocity_modes(ctx, p, g, redshift, t_rad, nblocks, st))) return rc;
  if ((rc = reduce_partials(ctx, ctx->partials, nblocks, 1, ctx->d_sums, st))) return rc;
  RG_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_sums, ctx->d_sums, sizeof(double), cudaMemcpyDeviceToHost, st));
  if (vel_modes && (rc = xy_ctrl_fetch(ctx, st))) return rc;
  RG_CUDA_TRY(ctx, cudaStreamSynchronize(st));
  if (vel_modes && (rc = xy_ctrl_result(ctx))) return rc;
  // the reference divides by N^3 before its Allreduce (BrightnessTemperature.c:528); on one rank
  // that is the same division
  *volume_ave_Tb = ctx->h_sums[0] / std::pow((double)n, 3);
  return RG_OK;
}

int rg_delta_T_host(rg_context* ctx, const rg_params* p, const rg_snapshot* s, const rg_grids* h,
                    double* volume_ave_Tb) {
  if (!ctx || !p || !s || !h || !volume_ave_Tb) return RG_EINVAL;
  if (p->ReionGridDim != ctx->N) return set_error(ctx, RG_EINVAL, "ReionGridDim differs from the context's grid");
  cudaSetDevice(ctx->device);
  if (!ctx->dev_grids_ready) {
    int rc = rg_alloc_grids(ctx, p, 0, &ctx->dev_grids);
    if (rc) return rc;
    ctx->dev_grids_ready = true;
  }
  const rg_grids& d = ctx->dev_grids;
  if (p->Flag_IncludeSpinTemp && !d.TS_box) return set_error(ctx, RG_EINVAL, "device grids lack TS_box");
  const size_t n = (size_t)ctx->N;
  const size_t bp = n * n * 2 * (n / 2 + 1) * sizeof(float), br = n * n * n * sizeof(float);
  cudaStream_t st = ctx->stream;
  RG_CUDA_TRY(ctx, cudaMemcpyAsync((void*)d.deltax, h->deltax, bp, cudaMemcpyHostToDevice, st));
  RG_CUDA_TRY(ctx, cudaMemcpyAsync(d.xH, h->xH, br, cudaMemcpyHostToDevice, st));
  if (p->Flag_IncludeSpinTemp) RG_CUDA_TRY(ctx, cudaMemcpyAsync(d.TS_box, h->TS_box, br, cudaMemcpyHostToDevice, st));
  rg_grids dv = d;
  if (p->Flag_IncludeSpinTemp && p->Flag_IncludePecVelsFor21cm > 0) {
    if (!h->vel) return set_error(ctx, RG_EINVAL, "missing grid pointer");
    int rv = ensure_device(ctx, &ctx->vel_stage, &ctx->vel_stage_elems, bp / sizeof(float));
    if (rv) return rv;
    RG_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->vel_stage, h->vel, bp, cudaMemcpyHostToDevice, st));
    dv.vel = ctx->vel_stage;
  }
  int rc = rg_delta_T(ctx, p, s, &dv, volume_ave_Tb);
  if (rc) return rc;
  RG_CUDA_TRY(ctx, cudaMemcpyAsync(h->delta_T, d.delta_T, br, cudaMemcpyDeviceToHost, st));
  RG_CUDA_TRY(ctx, cudaStreamSynchronize(st));
  return RG_OK;
}

}  // extern "C"
