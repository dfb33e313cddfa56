// The source grids from the galaxies, on the device: the nearest-grid-point deposit of
// construct_baryon_grids() (src/core/reionization.c:2025-2592) for one rank that holds the whole
// grid.  Every galaxy's values are added to the cell pos_to_ngp() (src/core/misc_tools.c:207-217)
// gives for its position; each grid is then clamped at zero (CLAMP_NEGATIVE, misc_tools.h:7),
// optionally divided (the sfr grid by the SFR timescale, reionization.c:2500-2510) and stored in
// the padded layout the steps read.  Which galaxy property feeds which grid, the black-hole mass
// limit and the shift of the history slots stay with the caller (the galaxy model).
//
// The reference adds a rank's galaxies to a float buffer in galaxy order; here the adds of the
// galaxies of one cell meet in any order (float atomics), which changes the cell sums by float
// rounding only.
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "rg_internal.h"
#include "rg_pass.cuh"

namespace rg {

constexpr int NGP_NT = 256;

// grid p of a pack without dynamic indexing into kernel parameters
__device__ __forceinline__ float* grid_of(const GridPtrsW& a, int p) {
  void* r = a.p[0];
#pragma unroll
  for (int i = 1; i < MAXG; ++i)
    if (p == i) r = a.p[i];
  return static_cast<float*>(r);
}

// pos_to_ngp: nearest grid point, the top edge wrapped to 0; -1 for a position below the box
__device__ __forceinline__ int ngp(float x, double side, int nx) {
  int ind = (int)rint((double)x / side * (double)nx);
  if (ind > nx - 1) ind = 0;
  return ind;
}

// zero the grids and the control words (npad floats each; npad is a multiple of 4, the base of a grid
// may not be)
__global__ void __launch_bounds__(NGP_NT) k_ngp_zero(GridPtrsW grids, size_t npad, int* __restrict__ ctrl) {
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 2) ctrl[threadIdx.x] = 0;
  float* g = grid_of(grids, blockIdx.y);
  const size_t step = (size_t)gridDim.x * NGP_NT, i0 = (size_t)blockIdx.x * NGP_NT + threadIdx.x;
  if (reinterpret_cast<uintptr_t>(g) % 16 == 0) {
    for (size_t i = i0; i < npad / 4; i += step) reinterpret_cast<float4*>(g)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  } else {
    for (size_t i = i0; i < npad; i += step) g[i] = 0.f;
  }
}

// ctrl[0]: galaxies below the box; ctrl[1]: bit p set when property p has a value below zero
__global__ void __launch_bounds__(NGP_NT) k_ngp_deposit(int n_gal, const float* __restrict__ pos, int n_prop,
                                                        const float* __restrict__ vals, GridPtrsW grids, double box,
                                                        int n, int* __restrict__ ctrl) {
  const int padw = 2 * (n / 2 + 1);
  int neg = 0;
  for (int g = blockIdx.x * NGP_NT + threadIdx.x; g < n_gal; g += gridDim.x * NGP_NT) {
    const int ix = ngp(pos[3 * (size_t)g], box, n), iy = ngp(pos[3 * (size_t)g + 1], box, n),
              iz = ngp(pos[3 * (size_t)g + 2], box, n);
    if (ix < 0 || iy < 0 || iz < 0) {
      atomicAdd(ctrl, 1);
      continue;
    }
    const size_t ip = ((size_t)ix * n + iy) * padw + iz;
    for (int p = 0; p < n_prop; ++p) {
      const float v = vals[(size_t)p * n_gal + g];
      if (v < 0.f) neg |= 1 << p;
      atomicAdd(grid_of(grids, p) + ip, v);
    }
  }
  if (neg) atomicOr(ctrl + 1, neg);
}

struct NgpDiv {
  double d[MAXG];
};

// clamp at zero and divide the cells of grid p0 + blockIdx.y (the padding holds zeros).  A grid whose values
// were all at least zero and whose divisor is 1 is final as it is: with the pass over it left out, and
// the others' in runs of 4, four grids of a 128^3 box and 10^6 galaxies took 82 us
// a call (145 before).
__global__ void __launch_bounds__(NGP_NT) k_ngp_finish(GridPtrsW grids, int p0, size_t npad, NgpDiv div,
                                                       const int* __restrict__ ctrl) {
  const int p = p0 + blockIdx.y;
  double dv = div.d[0];
#pragma unroll
  for (int i = 1; i < MAXG; ++i)
    if (p == i) dv = div.d[i];
  if (dv == 1.0 && !(ctrl[1] >> p & 1)) return;
  float* g = grid_of(grids, p);
  auto fin = [dv](float f) {
    double v = (double)f;
    if (v < 0) v = 0;
    return dv != 1.0 ? (float)(v / dv) : (float)v;
  };
  const size_t step = (size_t)gridDim.x * NGP_NT, i0 = (size_t)blockIdx.x * NGP_NT + threadIdx.x;
  if (reinterpret_cast<uintptr_t>(g) % 16 == 0) {
    for (size_t i = i0; i < npad / 4; i += step) {
      float4 v = reinterpret_cast<float4*>(g)[i];
      // most cells hold no galaxy
      if (v.x == 0.f && v.y == 0.f && v.z == 0.f && v.w == 0.f) continue;
      reinterpret_cast<float4*>(g)[i] = make_float4(fin(v.x), fin(v.y), fin(v.z), fin(v.w));
    }
  } else {
    for (size_t i = i0; i < npad; i += step) g[i] = fin(g[i]);
  }
}

}  // namespace rg

using namespace rg;

extern "C" {

int rg_deposit_ngp(rg_context* ctx, double box_size, int n_gal, const float* d_pos, int n_prop,
                   const float* d_values, const double* divisors, float* const* d_grids) {
  if (!ctx || !(box_size > 0) || n_gal < 0 || n_prop < 1 || !d_grids || (n_gal > 0 && (!d_pos || !d_values)))
    return RG_EINVAL;
  if (n_prop > MAXG) return set_error(ctx, RG_EINVAL, "at most 8 grids per deposit");
  cudaSetDevice(ctx->device);
  cudaStream_t st = ctx->stream;
  const int n = ctx->N;
  const size_t npad = (size_t)n * n * 2 * (n / 2 + 1);
  GridPtrsW gp{};
  NgpDiv dv;
  for (int p = 0; p < MAXG; ++p) dv.d[p] = 1.0;
  for (int p = 0; p < n_prop; ++p) {
    if (!d_grids[p]) return set_error(ctx, RG_EINVAL, "missing grid pointer");
    gp.p[p] = d_grids[p];
    if (divisors) {
      if (!(divisors[p] > 0)) return set_error(ctx, RG_EINVAL, "divisors must be positive");
      dv.d[p] = divisors[p];
    }
  }
  int rc = ensure_device(ctx, &ctx->ngp_bad, &ctx->ngp_bad_elems, 2);
  if (rc) return rc;
  const int nblk = 4 * ctx->num_sms;
  prof_begin(ctx, "ngp_zero", st);
  k_ngp_zero<<<dim3(nblk, n_prop), NGP_NT, 0, st>>>(gp, npad, ctx->ngp_bad);
  prof_end(ctx, 4.0 * n_prop * npad, st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  if (n_gal > 0) {
    prof_begin(ctx, "ngp_deposit", st);
    k_ngp_deposit<<<nblk, NGP_NT, 0, st>>>(n_gal, d_pos, n_prop, d_values, gp, box_size, n, ctx->ngp_bad);
    prof_end(ctx, (double)n_gal * (12.0 + 8.0 * n_prop), st);
    RG_CUDA_TRY(ctx, cudaGetLastError());
  }
  // properties that share a grid finish it one after the other, in their order
  bool shared = false;
  for (int p = 0; p < n_prop; ++p)
    for (int q = 0; q < p; ++q) shared = shared || gp.p[p] == gp.p[q];
  const int per = shared ? 1 : n_prop;
  prof_begin(ctx, "ngp_finish", st);
  for (int p = 0; p < n_prop; p += per) {
    k_ngp_finish<<<dim3(nblk, per), NGP_NT, 0, st>>>(gp, p, npad, dv, ctx->ngp_bad);
    RG_CUDA_TRY(ctx, cudaGetLastError());
  }
  prof_end(ctx, 8.0 * n_prop * (double)n * n * n, st);
  int bad = 0;
  RG_CUDA_TRY(ctx, cudaMemcpyAsync(&bad, ctx->ngp_bad, sizeof(int), cudaMemcpyDeviceToHost, st));
  RG_CUDA_TRY(ctx, cudaStreamSynchronize(st));
  if (bad) return set_error(ctx, RG_EINVAL, "galaxy positions below the box (pos_to_ngp asserts on them)");
  return RG_OK;
}

int rg_push_histories(rg_context* ctx, const rg_params* p, const rg_grids* g) {
  if (!ctx || !p || !g) return RG_EINVAL;
  if (!p->Flag_IncludeSpinTemp) return RG_OK;   // the reference keeps histories for ComputeTs only
  if (g->n_hist < 1) return set_error(ctx, RG_EINVAL, "n_hist must be at least 1");
  cudaSetDevice(ctx->device);
  cudaStream_t st = ctx->stream;
  const int n = ctx->N;
  const size_t npad = (size_t)n * n * 2 * (n / 2 + 1);
  const int agn = p->Flag_IncludeAGNXray;
  struct Kind {
    const float* cur;
    float* hist;
    bool on;
    const char* name;
  } kinds[4] = {  // the histories are inputs of the step (const in rg_grids); this call updates them
      {g->sfr, const_cast<float*>(g->sfr_histories), true, "sfr"},
      {g->xray_luminosity, const_cast<float*>(g->xray_luminosity_histories), true, "xray_luminosity"},
      {g->bh_xray_soft, const_cast<float*>(g->bh_xray_histories_soft), agn == 1 || agn == 3, "bh_xray_soft"},
      {g->bh_xray_hard, const_cast<float*>(g->bh_xray_histories_hard), agn == 1 || agn == 2, "bh_xray_hard"}};
  for (const Kind& k : kinds) {
    if (!k.on) continue;
    if (!k.cur || !k.hist) return set_error(ctx, RG_EINVAL, std::string("missing grid or histories of ") + k.name);
  }
  prof_begin(ctx, "push_histories", st);
  double bytes = 0.0;
  for (const Kind& k : kinds) {
    if (!k.on) continue;
    // slot h + 1 <- slot h from the top, then slot 0 <- this snapshot's grid
    for (int h = g->n_hist - 2; h >= 0; --h)
      RG_CUDA_TRY(ctx, cudaMemcpyAsync(k.hist + (size_t)(h + 1) * npad, k.hist + (size_t)h * npad,
                                       sizeof(float) * npad, cudaMemcpyDeviceToDevice, st));
    RG_CUDA_TRY(ctx, cudaMemcpyAsync(k.hist, k.cur, sizeof(float) * npad, cudaMemcpyDeviceToDevice, st));
    bytes += 8.0 * npad * g->n_hist;
  }
  prof_end(ctx, bytes, st);
  return RG_OK;
}

}  // extern "C"
