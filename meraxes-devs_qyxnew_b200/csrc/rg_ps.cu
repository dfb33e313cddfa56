// The callers next to the step on the output and input sides, on the library's transforms:
//
//   * the 21-cm power spectrum, Compute_PS() (src/core/ComputePowerSpectrum.c:44-255), which
//     dracarys.c:393-394 runs on delta_T right after ComputeBrightnessTemperatureBox(); its bin
//     count is Initialise_PowerSpectrum() (ComputePowerSpectrum.c:18-42);
//   * smooth_grid() (src/core/read_grids.c:127-165): forward transform, / N^3, real-space
//     top-hat of radius BoxSize / ReionGridDim / 2, inverse transform, applied to a grid read at
//     a finer resolution before it is subsampled.
//
// Power spectrum on the device: one pass sums delta_T (FP64 per block), one pass writes the
// padded real field ((delta_T / ave - 1) V / N^3) ave, the r2c transform (unnormalised, as
// FFTW's), then one pass over the Hermitian modes bins k^3 |delta_k|^2 / (2 pi^2 V), k and the
// mode count into per-block FP64 partials that the host adds in block order.  The modes' |k| and
// the bin edges are formed in float exactly as the reference does (products and sums rounded
// separately, the square root in double), so every mode lands in the reference's bin.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <vector>

#include "rg_internal.h"
#include "rg_pass.cuh"

namespace rg {

constexpr int PS_NT = 256;
constexpr int PS_MAXBINS = 64;

struct PsBins {
  float ceil[PS_MAXBINS];   // upper edge of bin i; its lower edge is ceil[i - 1] (0 for bin 0)
  int nb;
  float dk;                 // 2 pi / (BoxSize / h), float as in the reference
  double norm;              // 1 / (2 pi^2 V), V = powf(BoxSize / h, 3)
};

// the bin edges and count of Initialise_PowerSpectrum / Compute_PS (float arithmetic)
static PsBins ps_bins(const rg_params* p) {
  PsBins b;
  std::memset(&b, 0, sizeof(b));
  const double box_size = p->BoxSize / p->Hubble_h;  // Mpc
  const float k_factor = 1.35f;
  b.dk = (float)(2. * M_PI / box_size);
  const float k_max = b.dk * p->ReionGridDim;
  float k_ceil = b.dk;
  while (k_ceil < k_max && b.nb < PS_MAXBINS + 1) {
    if (b.nb < PS_MAXBINS) b.ceil[b.nb] = k_ceil;
    b.nb++;
    k_ceil *= k_factor;
  }
  const float volume = powf((float)box_size, 3);
  b.norm = 1.0 / (2.0 * M_PI * M_PI * (double)volume);
  return b;
}

__global__ void __launch_bounds__(PS_NT) k_ps_sum(const float* __restrict__ dT, size_t n3, double* partials) {
  double acc = 0.0;
  const size_t step = (size_t)gridDim.x * PS_NT;
  for (size_t i0 = (size_t)blockIdx.x * PS_NT + threadIdx.x; i0 < n3; i0 += 8 * step) {
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = i0 + k * step < n3 ? dT[i0 + k * step] : 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) acc += (double)v[k];
  }
  __shared__ double sh[PS_NT];
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int w = PS_NT / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) partials[blockIdx.x] = sh[0];
}

// deldel_ps (ComputePowerSpectrum.c:98-104) into a padded real grid; ave = sum / N^3 in double
__global__ void __launch_bounds__(PS_NT) k_ps_prepare(const float* __restrict__ dT, int n, const double* __restrict__ sum,
                                                      float volume, float* __restrict__ pad) {
  const size_t total = (size_t)n * n * n, step = (size_t)gridDim.x * PS_NT;
  const double n3 = (double)n * n * n;
  const double ave = *sum / n3, inv_ave = 1.0 / ave, f = (double)volume / (double)(float)n3;
#pragma unroll 4
  for (size_t i = (size_t)blockIdx.x * PS_NT + threadIdx.x; i < total; i += step) {
    const float v = (float)(((double)dT[i] * inv_ave - 1) * f);
    pad[i + ((unsigned)i / (unsigned)n) * 2] = (float)((double)v * ave);   // rows of n + 2 values
  }
}

// |k| of mode (nx, ny, nz) as Compute_PS forms it: float components, float squares and sums
// (no contraction), the square root rounded to float
__device__ __forceinline__ float ps_kmag(int nx, int ny, int nz, int n, float dk) {
  const int h = n / 2;
  const float kx = (float)(nx > h ? nx - n : nx) * dk;
  const float ky = (float)(ny > h ? ny - n : ny) * dk;
  const float kz = (float)nz * dk;
  const float s = __fadd_rn(__fadd_rn(__fmul_rn(kx, kx), __fmul_rn(ky, ky)), __fmul_rn(kz, kz));
  return __fsqrt_rn(s);   // the float nearest the root, as the C's (float)sqrt((double)s)
}

// per-block sums [3][nb]: k^3 |d|^2 norm, k, count over the Hermitian modes S[kz][x][y].  A thread
// walks x at its own (kz, y), a block taking xc values of x and PS_NT columns (kz, y) at a time: its
// bin changes a few times in a walk, so it sums in registers and adds to the block's shared sums when
// the bin changes (an FP64 add in shared memory is a compare-and-swap loop; one per mode or warp took
// 0.34 ms at 256^3, now 0.09).
constexpr int PS_XC = 64;   // the longest walk

// The longest walk that still gives two blocks an SM.  us with walks of 64 and by this rule: 16^3 38, 16;
// 64^3 85, 28; 96^3 89, 31; 128^3 80, 35; 192^3 81, 56 (walks of 2 at 256^3: 352 against 87).
static int ps_walk(int n, int num_sms) {
  const int groups = ((n / 2 + 1) * n + PS_NT - 1) / PS_NT;
  int xc = PS_XC;
  while (xc > 2 && groups * ((n + xc - 1) / xc) < 2 * num_sms) xc /= 2;
  return xc;
}

__global__ void __launch_bounds__(PS_NT) k_ps_bins(const cf* __restrict__ spec, int n, int xc, const PsBins b,
                                                   double* __restrict__ partials) {
  __shared__ double sums[3][PS_MAXBINS];
  __shared__ float ceil_s[PS_MAXBINS];
  for (int i = threadIdx.x; i < PS_MAXBINS; i += PS_NT) {
    sums[0][i] = sums[1][i] = sums[2][i] = 0.0;
    ceil_s[i] = i < b.nb ? b.ceil[i] : 0.f;
  }
  __syncthreads();
  const int nb = max(b.nb, 1);
  const size_t cols = (size_t)(n / 2 + 1) * n;   // (kz, y), y fastest
  const size_t groups = (cols + PS_NT - 1) / PS_NT, chunks = (n + xc - 1) / xc;
  for (size_t w = blockIdx.x; w < groups * chunks; w += gridDim.x) {
    const size_t col = w / chunks * PS_NT + threadIdx.x;
    if (col >= cols) continue;
    const int y = (int)(col % n), kz = (int)(col / n);
    const int x0 = (int)(w % chunks) * xc, x1 = min(n, x0 + xc);
    int bin = -1;
    double pw = 0.0, kk = 0.0;
    int cnt = 0;
    auto flush = [&] {
      if (bin >= 0 && cnt) {
        atomicAdd(&sums[0][bin], pw * b.norm);
        atomicAdd(&sums[1][bin], kk);
        atomicAdd(&sums[2][bin], (double)cnt);
      }
      pw = kk = 0.0;
      cnt = 0;
    };
    const float2* src = reinterpret_cast<const float2*>(spec + (size_t)kz * n * n + y);
#pragma unroll 4
    for (int x = x0; x < x1; ++x) {
      const float2 v = __ldg(src + (size_t)x * n);
      const float km = ps_kmag(x, y, kz, n, b.dk);
      // the first bin whose upper edge exceeds |k| (bins are contiguous from 0)
      int nbin = bin;
      if (!(bin >= 0 && km < ceil_s[bin] && (bin == 0 || !(km < ceil_s[bin - 1])))) {
        nbin = -1;
        if (km < ceil_s[nb - 1]) {
          nbin = 0;
          while (!(km < ceil_s[nbin])) ++nbin;
        }
      }
      if (nbin != bin) {
        flush();
        bin = nbin;
      }
      const double kd = (double)km;
      pw += kd * kd * kd * ((double)v.x * v.x + (double)v.y * v.y);
      kk += kd;
      cnt += 1;
    }
    flush();
  }
  __syncthreads();
  double* out = partials + (size_t)blockIdx.x * 3 * PS_MAXBINS;
  for (int i = threadIdx.x; i < 3 * PS_MAXBINS; i += PS_NT) out[i] = sums[i / PS_MAXBINS][i % PS_MAXBINS];
}

static int power_spectrum(rg_context* ctx, const rg_params* p, const float* d_dT, int max_bins, float* PS_k,
                          float* PS_data, float* PS_error, int* n_bins) {
  int rc = validate_common(ctx, p);
  if (rc) return rc;
  if (!(p->Hubble_h > 0)) return set_error(ctx, RG_EINVAL, "Hubble_h must be positive");
  const PsBins b = ps_bins(p);
  if (b.nb > PS_MAXBINS) return set_error(ctx, RG_EUNSUPPORTED, "more than 64 power-spectrum bins");
  *n_bins = b.nb;
  if (max_bins < b.nb) return set_error(ctx, RG_EINVAL, "max_bins is smaller than the number of bins");
  cudaStream_t st = ctx->stream;
  const int N = ctx->N;
  const size_t n3 = (size_t)N * N * N, nc = (size_t)(N / 2 + 1) * N * N, npad = 2 * nc;
  if ((rc = ensure_device(ctx, &ctx->spec, &ctx->spec_elems, nc))) return rc;
  if ((rc = ensure_device(ctx, &ctx->ps_pad, &ctx->ps_pad_elems, npad))) return rc;
  const int nblk = 4 * ctx->num_sms;
  double* partials = ensure_partials(ctx, (size_t)nblk * 3 * PS_MAXBINS);
  if (!partials) return set_error(ctx, RG_ENOMEM, "partials");
  const double box_size = p->BoxSize / p->Hubble_h;
  const float volume = powf((float)box_size, 3);

  prof_begin(ctx, "ps_sum", st);
  k_ps_sum<<<nblk, PS_NT, 0, st>>>(d_dT, n3, partials);
  prof_end(ctx, 4.0 * n3, st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  if ((rc = reduce_partials(ctx, partials, nblk, 1, ctx->d_sums, st))) return rc;
  prof_begin(ctx, "ps_prepare", st);
  k_ps_prepare<<<nblk, PS_NT, 0, st>>>(d_dT, N, ctx->d_sums, volume, ctx->ps_pad);
  prof_end(ctx, 8.0 * n3, st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  const float* src = ctx->ps_pad;
  if ((rc = fft_forward(ctx, N, &src, 1, ctx->spec, nc, 1.0, st))) return rc;
  prof_begin(ctx, "ps_bins", st);
  k_ps_bins<<<nblk, PS_NT, 0, st>>>(ctx->spec, N, ps_walk(N, ctx->num_sms), b, partials);
  prof_end(ctx, 8.0 * nc, st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  std::vector<double> h((size_t)nblk * 3 * PS_MAXBINS);
  RG_CUDA_TRY(ctx, cudaMemcpyAsync(h.data(), partials, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, st));
  RG_CUDA_TRY(ctx, cudaStreamSynchronize(st));
  prof_resolve(ctx);
  for (int i = 0; i < b.nb; ++i) {
    double pbox = 0.0, kave = 0.0, cnt = 0.0;
    for (int k = 0; k < nblk; ++k) {
      const double* q = h.data() + (size_t)k * 3 * PS_MAXBINS;
      pbox += q[i];
      kave += q[PS_MAXBINS + i];
      cnt += q[2 * PS_MAXBINS + i];
    }
    // ComputePowerSpectrum.c:233-235 (an empty bin gives 0/0, as there)
    PS_k[i] = (float)(kave / cnt);
    PS_data[i] = (float)(pbox / cnt);
    PS_error[i] = (float)((pbox / cnt) / sqrt(cnt));
  }
  return RG_OK;
}

}  // namespace rg

using namespace rg;

extern "C" {

int rg_power_spectrum_length(const rg_params* p, int* n_bins) {
  if (!p || !n_bins || p->ReionGridDim <= 0 || !(p->BoxSize > 0) || !(p->Hubble_h > 0)) return RG_EINVAL;
  *n_bins = ps_bins(p).nb;
  return RG_OK;
}

int rg_power_spectrum(rg_context* ctx, const rg_params* p, const float* d_delta_T, int max_bins, float* PS_k,
                      float* PS_data, float* PS_error, int* n_bins) {
  if (!ctx || !p || !d_delta_T || !PS_k || !PS_data || !PS_error || !n_bins) return RG_EINVAL;
  cudaSetDevice(ctx->device);
  return power_spectrum(ctx, p, d_delta_T, max_bins, PS_k, PS_data, PS_error, n_bins);
}

int rg_power_spectrum_host(rg_context* ctx, const rg_params* p, const float* h_delta_T, int max_bins, float* PS_k,
                           float* PS_data, float* PS_error, int* n_bins) {
  if (!ctx || !p || !h_delta_T || !PS_k || !PS_data || !PS_error || !n_bins) return RG_EINVAL;
  int rc = validate_common(ctx, p);
  if (rc) return rc;
  cudaSetDevice(ctx->device);
  const size_t n3 = (size_t)ctx->N * ctx->N * ctx->N;
  if ((rc = ensure_device(ctx, &ctx->ps_stage, &ctx->ps_stage_elems, n3))) return rc;
  RG_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->ps_stage, h_delta_T, sizeof(float) * n3, cudaMemcpyHostToDevice, ctx->stream));
  return power_spectrum(ctx, p, ctx->ps_stage, max_bins, PS_k, PS_data, PS_error, n_bins);
}

int rg_smooth_grid(rg_context* ctx, double box_size, int reion_grid_dim, const float* d_in_padded,
                   float* d_out_padded) {
  if (!ctx || !d_in_padded || !d_out_padded || !(box_size > 0) || reion_grid_dim <= 0) return RG_EINVAL;
  cudaSetDevice(ctx->device);
  rg_params p;
  // the grid being smoothed is the context's (read_grids.c passes its n_cell)
  if (rg_params_default(&p, ctx->N, box_size) != RG_OK) return RG_EINVAL;
  // read_grids.c:151-155: float radius, real-space top-hat
  const double R = (double)(float)(box_size / (double)reion_grid_dim / 2.0);
  int rc = debug_roundtrip(ctx, &p, d_in_padded, d_out_padded, R, 0);
  if (rc) return rc;
  RG_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  return RG_OK;
}

}  // extern "C"
