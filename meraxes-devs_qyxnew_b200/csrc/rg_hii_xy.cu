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
#define RG_XY(PLAN, BL) launch_xy_fused<N, PLAN<N>, BL>(ctx, op, spec, ng, nr, "inv_xy_c2c_window", bytes, st)
    // Where 3 divides N, the plan over more threads a line (PlanZ: 12 values a thread at most; PlanW: 24): always
    // while its lines take up to 8 threads; with up to 32 (a warp) from 4 grids an item on, at three blocks
    // an SM (PlanW's registers spill there), or two where the planes that three have in flight would not stay
    // in L2; with 64, blocks of 512, never.  2, 3, 4, 6, 8, 12 grids an item, PlanW then PlanZ:
    //   24^3    44 52 61 78 94 130          40 44 47 60 65 81 us
    //   48^3    101 129 168 246 323 459     74 87 104 134 167 246 us
    //   96^3    288 410 545 901 1225 1909   at two blocks 405 509 616 827 1042 1494, at three 330 425 524 720 939 1481 us
    //   192^3   1.84 2.72 4.78 7.92 10.8 16.4   3.14 4.01 4.89 6.67 8.50 12.3, 2.61 3.44 4.30 6.09 8.05 12.4 ms
    //   384^3   14.1 21.4 33.6 51.4         29.3 39.0 48.8 69.0 ms
    // and with the sharp-k window, 8 and 12 grids at two and three blocks: 96^3 983 902, 1432 1489 us; 192^3 8.07 7.85,
    // 11.8 12.8 ms.
    if constexpr (N % 3 == 0 && PlanZ<N>::T <= 32) {
      if constexpr (PlanZ<N>::T <= 8) return RG_XY(PlanZ, 2);
      if (ng >= 4)
        return xy_least_planes<N, PlanZ<N>, 3>(ctx, ng) <= XY_PLANES ? RG_XY(PlanZ, 3) : RG_XY(PlanZ, 2);
    }
    // Powers of two: three blocks an SM for 2 grids an item, two for more, whose planes in flight do not stay in
    // L2 with the third.  us for 2, 3, 4, 6 grids, two blocks then three:
    //   64^3    90 115 138 186         87 112 136 198
    //   128^3   470 650 831 1304       474 653 832 1308
    //   256^3   3.04 4.20 5.37 9.00    2.89 4.42 7.24 12.6 (ms)
    //   512^3   31.6 44.7 - -          33.5 47.3 - -       (ms; its registers spill at three)
    // (Smaller boxes have no blocks of 256 threads.)
    if constexpr (N % 3 != 0 && PlanW<N>::T <= 16 && XYF<N, PlanW<N>, 2>::NTH == 256)
      if (ng <= 2) return RG_XY(PlanW, 3);
    return RG_XY(PlanW, 2);
#undef RG_XY
  }
  if (ngu != ng) return set_error(ctx, RG_EINVAL, "several snapshots in one pass need the fused mode");
  return launch_win_xy<N>(ctx, op, spec, stride, ng, nr, st);
}

int inverse_xy(rg_context* ctx, int n, const cf* spec, int ng, int ngu, cf* work, size_t stride, int nr,
                      const float* wplanes, int unfiltered, cudaStream_t st, const int* wcut) {
  RG_DISPATCH_N(n, launch_inverse_xy<NN>(ctx, spec, ng, ngu, work, stride, nr, wplanes, unfiltered, st, wcut));
}

}  // namespace rg
