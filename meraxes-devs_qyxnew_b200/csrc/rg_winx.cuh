// The windowed inverse x pass of a batch of radii: every grid's spectrum times the window of each
// radius of the batch, transformed along x into the work buffer (the y pass follows in place).
#pragma once

#include "rg_internal.h"
#include "rg_pass.cuh"

namespace rg {

template <int N>
struct WinX {
  using PL = PlanW<N>;
  static constexpr int T = PL::T;
  static constexpr int V = N / T;
  static constexpr int B = Cfg<N>::BX;   // columns of a block
  static constexpr int NTH = T * B;
  static constexpr int MINB = NTH >= 512 ? 1 : NTH >= 256 ? 3 : NTH >= 128 ? 5 : 8;
  static constexpr size_t smem() { return sizeof(cf) * (N + (size_t)line_buf_r0<N, PL::R[0], B>()); }
};

template <int N, class Op>
__global__ void __launch_bounds__(WinX<N>::NTH, WinX<N>::MINB)
    k_win_x(Op op, int nr, const cf* __restrict__ spec, size_t stride, const cf* __restrict__ g_tw) {
  using W = WinX<N>;
  using PL = typename W::PL;
  constexpr int B = W::B, V = W::V, WP = wplane_pitch(N);
  extern __shared__ cf smem[];
  cf* s_tw = smem;
  cf* xbuf = smem + N;
  const int kz = blockIdx.y;
  const int b = threadIdx.x % B, t = threadIdx.x / B;
  const int y = blockIdx.x * B + b, ny = y > N / 2 ? N - y : y;
  const size_t col = (size_t)kz * N * N + y;
  load_twiddles_p<PL>(s_tw, g_tw);
  __syncthreads();
  const int ng = op.grids();
  for (int r = 0; r < nr; ++r) {
    float wv[V];
    const bool fil = op.filtered(r);
    const int cut = op.cutoff(r);
    const float* wp = op.wplane(r) + (size_t)kz * (N / 2 + 1) * WP + ny;
#pragma unroll
    for (int sl = 0; sl < V; ++sl) {
      const int p = stage0_pos<PL>(t, sl);
      const int nx = p > N / 2 ? N - p : p;
      wv[sl] = !fil ? 1.f : cut >= -1 ? (nx * nx + ny * ny + kz * kz <= cut ? 1.f : 0.f) : __ldg(wp + nx * WP);
    }
    for (int g = 0; g < ng; ++g) {
      const cf* src = spec + (size_t)g * stride + col;
      cf* dst = op.out(r, g) + col;
      line_fft_p<PL, true>(
          t, xbuf, s_tw,
          [&](int p, int sl) {
            const float2 v = __ldg(reinterpret_cast<const float2*>(src + (size_t)p * N));
            return cf{v.x * wv[sl], v.y * wv[sl]};
          },
          [&](int p) { return line_addr_r0<PL::R[0], B>(p, b); },
          [&](int p, cf v, int) { dst[(size_t)p * N] = v; });
    }
  }
}

template <int N, class Op>
int launch_win_xy(rg_context* ctx, const Op& op, const cf* spec, size_t stride, int ng, int nr, cudaStream_t st) {
  using W = WinX<N>;
  const cf* tw;
  int rc = twiddles_for(ctx, N, &tw);
  if (rc) return rc;
  const double nzc = (double)Cfg<N>::NZ * N * N;
  auto kern = k_win_x<N, Op>;
  RG_CUDA_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)W::smem()));
  prof_begin(ctx, "inv_x_c2c_window", st);
  kern<<<dim3(N / W::B, Cfg<N>::NZ), W::NTH, W::smem(), st>>>(op, nr, spec, stride, tw);
  prof_end(ctx, ng * 8.0 * nzc * (1 + nr), st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  prof_begin(ctx, "inv_y_c2c", st);
  RG_CUDA_TRY(ctx, (launch_pass_y<N, true>(op.work, stride, ng * nr, tw, st)));
  prof_end(ctx, ng * nr * 16.0 * nzc, st);
  return RG_OK;
}

}  // namespace rg
