// The windowed inverse x and y passes of find_HII_bubbles.
#include <cuda_runtime.h>

#include <string>

#include "rg_internal.h"
#include "rg_pass.cuh"
#include "rg_tma.cuh"
#include "rg_winx.cuh"
#include "rg_xyf.cuh"

namespace rg {

// the batch of the fused x/y pass: grid g of spec windowed for radius r into work (r ng + g)
// The grids may be several snapshots' (ngu grids each, the same radii): the work buffer holds
// snapshot u's block [radius][its grids] at u nr ngu (one snapshot: [radius][grid]).
struct HiiXOp {
  const cf* spec;
  size_t stride;
  int ng;
  int ngu;           // grids per snapshot
  int nr;            // radii of the batch
  cf* work;
  const float* wplanes;
  size_t wsize;      // one radius's window
  int unfiltered;
  const int* wcut;   // sharp-k step ends per radius, or null (the planes are read)
  __device__ int grids() const { return ng; }
  __device__ bool filtered(int r) const { return r != unfiltered; }
  __device__ const float* wplane(int r) const { return wplanes + (size_t)r * wsize; }
  __device__ int cutoff(int r) const { return wcut ? __ldg(wcut + r) : -2; }
  __device__ cf* out(int r, int g) const {
    const int u = g / ngu;
    return work + (((size_t)u * nr + r) * ngu + (g - u * ngu)) * stride;
  }
};

// inverse x (window, batch of nr radii) and y passes: one fused kernel, or (plain mode) the two
// passes as separate kernels
template <int N>
int launch_inverse_xy(rg_context* ctx, const cf* spec, int ng, int ngu, cf* work, size_t stride, int nr,
                      const float* wplanes, int unfiltered, cudaStream_t st, const int* wcut = nullptr) {
  using C = Cfg<N>;
  const double nzc = (double)C::NZ * N * N;
  const HiiXOp op{spec, stride, ng, ngu, nr, work, wplanes, wplane_size(N), unfiltered, wcut};
  if (ctx->mode == RG_MODE_FUSED) {
    if (stride != (size_t)C::NZ * N * N) return set_error(ctx, RG_EINVAL, "fused x/y pass: spectra must be contiguous");
    const double bytes = ng * 8.0 * nzc * (1 + nr);
    // 96^3: the plan over 16 threads a line from 6 grids an item (several snapshots) on, 1.5 against 2.1
    // ms for 12 grids; its smaller items cost more with the 2 or 3 grids of one (0.40 against 0.29 ms)
    if constexpr (N == 96)
      if (ng >= 6) return launch_xy_fused<N, PlanZ<N>>(ctx, op, spec, ng, nr, "inv_xy_c2c_window", bytes, st);
    return launch_xy_fused<N, PlanW<N>>(ctx, op, spec, ng, nr, "inv_xy_c2c_window", bytes, st);
  }
  if (ngu != ng) return set_error(ctx, RG_EINVAL, "several snapshots in one pass need the fused mode");
  return launch_win_xy<N>(ctx, op, spec, stride, ng, nr, st);
}

int inverse_xy(rg_context* ctx, int n, const cf* spec, int ng, int ngu, cf* work, size_t stride, int nr,
                      const float* wplanes, int unfiltered, cudaStream_t st, const int* wcut) {
  RG_DISPATCH_N(n, launch_inverse_xy<NN>(ctx, spec, ng, ngu, work, stride, nr, wplanes, unfiltered, st, wcut));
}

}  // namespace rg
