// Forward r2c transforms of the step's grids.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "rg_internal.h"
#include "rg_pass.cuh"

namespace rg {

template <typename K>
static cudaError_t prep(K kernel, size_t smem) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

template <int N>
constexpr size_t smem_x() { return sizeof(cf) * (N + (size_t)line_buf<N, Cfg<N>::BX>()); }

template <int N>
int launch_forward(rg_context* ctx, const float* const* d_real, int ng, cf* spec, size_t stride, double scale,
                   cudaStream_t st) {
  const cf* tw;
  int rc = twiddles_for(ctx, N, &tw);
  if (rc) return rc;
  using C = Cfg<N>;
  FwdSrcs src{};
  for (int g = 0; g < ng; ++g) src.p[g] = d_real[g];
  const double nzc = (double)C::NZ * N * N;
  using ZF = ZFCfg<N>;
  RG_CUDA_TRY(ctx, prep(k_fwd_z<N>, ZF::smem()));
  prof_begin(ctx, "fwd_z_r2c", st);
  k_fwd_z<N><<<dim3(N / (2 * ZF::QF), N, ng), ZF::NTH, ZF::smem(), st>>>(src, spec, stride, tw);
  prof_end(ctx, ng * (4.0 * N * N * N + 8.0 * nzc), st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  prof_begin(ctx, "fwd_y_c2c", st);
  RG_CUDA_TRY(ctx, (launch_pass_y<N, false>(spec, stride, ng, tw, st)));
  prof_end(ctx, ng * 16.0 * nzc, st);
  RG_CUDA_TRY(ctx, prep((k_pass_x<N, false>), smem_x<N>()));
  prof_begin(ctx, "fwd_x_c2c", st);
  k_pass_x<N, false><<<dim3(N / C::BX, C::NZ, ng), C::T * C::BX, smem_x<N>(), st>>>(spec, stride, tw, (float)scale);
  prof_end(ctx, ng * 16.0 * nzc, st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  return RG_OK;
}

// Grids a forward launch takes: as many as L2 holds between the three passes (64 MB of it), 8 at least.
// 56 grids at 64^3 (ComputeTs, with its frequency integrals running beside): 82 us in one launch of each
// pass, 203 in seven.
int fft_forward_group(int n) {
  const double bytes = 8.0 * (n / 2 + 1) * n * n;
  return std::min(FWD_MAXG, std::max(MAXG, (int)(64.0 * 1024 * 1024 / bytes)));
}

int fft_forward(rg_context* ctx, int n, const float* const* d_real, int ng, cf* spec, size_t stride, double scale,
                cudaStream_t st) {
  if (ng > FWD_MAXG) return set_error(ctx, RG_EINVAL, "too many grids in one forward launch");
  RG_DISPATCH_N(n, launch_forward<NN>(ctx, d_real, ng, spec, stride, scale, st));
}

}  // namespace rg
