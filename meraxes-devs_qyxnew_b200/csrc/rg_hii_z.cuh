// The z pass of find_HII_bubbles: per-snapshot constants and state, and the kernel k_hii_zr (c2r along
// z from tensor tiles, barrier test on the transform's registers).  rg_hii.cu holds the row-buffer
// form for Pop III sources and small boxes, the closing pass and the snapshot itself.
#pragma once

#include <math.h>

#include <string>
#include <type_traits>
#include <utility>

#include "rg_internal.h"
#include "rg_pass.cuh"
#include "rg_tma.cuh"

namespace rg {

struct HiiBatch {
  int nr;             // radii in this batch
  int first;          // the batch starts the snapshot (state comes from z_at_ionization)
  int last;           // the batch ends with the snapshot's last (unfiltered) radius
  int ng;             // grids per radius (k_hii_zr and the plain forms of k_hii_z know it at compile time)
  double fcoll_pref[KB_MAX];
  float J_aux[KB_MAX], J_aux_bh[KB_MAX];
  float G_pref[KB_MAX], G_pref_bh[KB_MAX], R[KB_MAX];   // recombination branch
};

// the same for Pop III sources (mini-halos)
struct HiiBatchIII {
  double fcoll_pref[KB_MAX];
  float J_aux[KB_MAX], G_pref[KB_MAX];
};

struct HiiState {
  float* xH;
  float* z_in;
  float* J21;
  float* temp;
  const float* Tk_box;
  const float* deltax_unf;   // padded
  const float* wsfr;         // padded
  const float* bhar;         // padded, may be null
  const float* wsfrIII;      // padded, Pop III only
  float* Gamma12;            // recombination branch: written at a cell's first crossing
  float* r_bubble;
  // between radius batches, per cell: z_at_ionization still < 0 (A); ionised at a radius of this
  // snapshot (I).  k_hii_zr keeps a thread's cells as two words, k_hii_z a byte per cell (A + 2 I).
  uint8_t* state;
};


// one snapshot of a z pass; several independent ones share a launch (blockIdx.z)
struct HiiZUnit {
  HiiBatch bt;
  HiiConst c;
  HiiState s;
};
constexpr int HII_ZU = 8;
struct HiiZUnits {
  HiiZUnit u[HII_ZU];
};

// f(std::integral_constant<int, I>{}) for I in the sequence, in order
template <class F, int... I>
__device__ __forceinline__ void for_each_index(std::integer_sequence<int, I...>, F&& f) {
  (f(std::integral_constant<int, I>{}), ...);
}

// ---------------------------------------------------------------------------
// z pass of a batch, with the tiles staged by TMA and the barrier test on the transforms' registers.
//
// The block owns rows [y0, y0 + 2Q) of plane x.  For every (radius, grid) unit of the batch, the
// Hermitian half column tile (all kz, those rows) arrives in shared memory by tensor loads (ZB
// tiles in flight, one mbarrier each); the c2r of its row pairs leaves each thread the same cells
// of every grid (the transform's output positions do not depend on the grid), so the previous
// grids' values are kept in registers and the clamp and barrier test run as the last tested grid's
// values come out of the transform: no row buffer in shared memory.  The state of a cell
// (z_at_ionization still < 0; ionised at a radius of this snapshot) is two bits in registers
// within the batch and in a word per thread between batches.  At the snapshot's last radius it
// writes xH, negative (or -0) where the cell was neutral at every radius: the closing pass
// (k_hii_close) takes it from there.
//
// It is bound by its own instructions at the occupancy its registers allow, so the sizes with a
// factor 3 run their plans over more threads (PlanZ): 12 cells a thread instead of 48.  The rare
// writes and the closing radius' divisions stay out of the test's code, which fits the instruction
// cache then.  z passes of a snapshot with its closing pass, before (row buffers at the sizes with a
// factor 3 and for recombinations, closing pass inside) and now: 192^3 47 radii 3 grids 4.52 -> 1.46
// ms, 6 x 96^3 3.17 -> 0.78, 128^3 with recombinations 1.47 -> 1.05, 256^3 2.91 -> 1.92, 512^3 39.8 ->
// 33.2.
template <int N>
struct HiiZR {
  static constexpr bool USED = N >= 64;   // the smaller boxes take the row-buffer form
  using PL = PlanZ<N>;
  static constexpr int T = PL::T, Q = pow2_div(N / 2, cmax(128 / T, 4)), NTH = T * Q;
  static constexpr int VL = last_values<PL>();   // z values of a row a thread ends with
  static constexpr int NZ = N / 2 + 1;
  // kz rows per tensor box (box dimensions are at most 256): one box, or for N = 512 two boxes of
  // (NZ + 1) / 2 rows at kz 0 and kz NZ - KZB that overlap in one row, so the second box lands on
  // a 128-byte boundary of the tile and no row lies outside the tensor
  static constexpr int KZB = NZ <= 256 ? NZ : (NZ + 1) / 2;
  static constexpr int NBOX = NZ <= 256 ? 1 : 2;
  static constexpr int TB = round_up(cmax(NZ * 2 * Q, line_buf<N, Q>()), 16);   // 128-byte multiple
  static constexpr int ZB = 3;                                 // tiles in flight
  static constexpr uint32_t TX = (uint32_t)(NBOX * KZB * 2 * Q * sizeof(cf));   // bytes the boxes deliver
  static_assert(NBOX == 1 || ((NZ - KZB) * 2 * Q * sizeof(cf)) % 128 == 0, "second box off a 128-byte boundary");
  static constexpr size_t smem() { return 128 + sizeof(cf) * ((size_t)ZB * TB + N) + sizeof(uint64_t) * ZB; }
  // resident blocks: register room for the KEPT values a thread keeps of the grids before the last
  // tested one, without spills
  template <int KEPT>
  static constexpr int minb() {
    if (NTH >= 256) return KEPT > 32 ? 1 : 2;
    if (VL <= 8) return KEPT > 24 ? 3 : KEPT > 16 ? 4 : 5;
    return KEPT > 64 ? 2 : 3;
  }
  // the batch runs' sizes take several snapshots a launch; one alone fills the chip above them, and
  // a fixed index keeps its constants in instruction operands (2.0 against 2.2 ms at 256^3)
  static constexpr bool MULTI = N <= 128;
  using Word = std::conditional_t<(2 * VL <= 16), uint16_t, uint32_t>;   // a thread's A or I bits
  static_assert(2 * VL <= 32, "a thread's state bits in one word");
  static_assert((N / PL::R[PL::S - 1]) % T == 0, "every thread ends with VL values");
};

constexpr int TMA_WAIT_LIMIT = 1 << 22;   // polls of an mbarrier before a wait gives up

// Grids per radius: deltax, stars, [x_e], [effective_bhm], [N_rec], tested; with REC then weighted_sfr
// and with BH effective_bhar, which give Gamma12 where a cell first crosses.
//
// FINAL: the batch ends with the snapshot's last radius (the code of its partial xH, 2 VL divisions
// long, stays out of the other batches' instruction cache).
template <int N, bool SPIN, bool BH, bool REC, bool FINAL>
__global__ void __launch_bounds__(HiiZR<N>::NTH,
                                  (HiiZR<N>::template minb<(1 + SPIN + BH + REC) * 2 * HiiZR<N>::VL>()))
    k_hii_zr(const __grid_constant__ CUtensorMap tmap, const cf* __restrict__ g_tw,
             const __grid_constant__ HiiZUnits us, uint32_t* err) {
  using Z = HiiZR<N>;
  using PL = typename Z::PL;
  constexpr int Q = Z::Q, VL = Z::VL, ZB = Z::ZB, TB = Z::TB, NZ = Z::NZ, KZB = Z::KZB, NBOX = Z::NBOX;
  using Word = typename Z::Word;
  constexpr int NT = 2 + SPIN + BH + REC;                    // tested grids
  constexpr int NG = NT + (REC ? 1 + BH : 0);
  [[maybe_unused]] constexpr int GX = 2, GB = 2 + SPIN, GN = 2 + SPIN + BH;   // x_e, effective_bhm, N_rec
  const HiiZUnit& un = us.u[Z::MULTI ? blockIdx.z : 0];
  const HiiBatch& bt = un.bt;
  const HiiConst& c = un.c;
  const HiiState& s = un.s;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  cf* tiles = reinterpret_cast<cf*>(sm);
  cf* s_tw = tiles + ZB * TB;
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_tw + N);
  const int x = blockIdx.y, y0 = blockIdx.x * 2 * Q;
  const int q = threadIdx.x % Q, tq = threadIdx.x / Q;
  const int nunits = bt.nr * NG;
  const int spec0 = Z::MULTI ? blockIdx.z * nunits : 0;   // this snapshot's first spectrum

  if (threadIdx.x == 0) {
    for (int b = 0; b < ZB; ++b) mbar_init(&bars[b], 1);
    mbar_init_fence();
  }
  load_twiddles_p<PL>(s_tw, g_tw);
  __syncthreads();
  // thread 0: tensor loads of unit u into tile u % ZB (tensor coordinates: y in floats, x, kz of
  // the unit's spectrum stacked after the previous units)
  auto issue = [&](int u) {
    const int b = u % ZB;
    mbar_arrive_expect_tx(&bars[b], Z::TX);
#pragma unroll
    for (int k = 0; k < NBOX; ++k) {
      const int k0 = k ? NZ - KZB : 0;
      tma_load_3d(tiles + b * TB + k0 * 2 * Q, &tmap, 2 * y0, x, (spec0 + u) * NZ + k0, &bars[b]);
    }
  };
  if (threadIdx.x == 0)
    for (int u = 0; u < ZB && u < nunits; ++u) issue(u);

  // state of this thread's 2 VL cells: cell 2 slot + h is row y0 + 2q + h at z = last_pos(tq, slot)
  uint32_t A = 0, I = 0;
  uint32_t X = 0;   // REC: first crossing of the snapshot at the radius in work
  Word* state = reinterpret_cast<Word*>(s.state) +
                2 * (((size_t)blockIdx.y * gridDim.x + blockIdx.x) * Z::NTH + threadIdx.x);
  if (bt.first) {
#pragma unroll
    for (int slot = 0; slot < VL; ++slot) {
      const int z = last_pos<PL>(tq, slot);
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (s.z_in[((size_t)x * N + y0 + 2 * q + h) * N + z] < 0.f) A |= 1u << (2 * slot + h);
    }
  } else {
    A = state[0];
    I = state[1];
  }

  float vals[NT][2 * VL];   // the tested grids at the radius in work
  // the clamped fields of this thread's cell k and its neutral share nf; returns N_rec / (1 + delta)
  auto clamped = [&](int k, float* st_out, float* bhm_out, double* dom_out, double* nf_out) -> double {
    const float dx = fmaxf(vals[0][k], -1.f + REL_TOL);
    float st = fmaxf(vals[1][k], 0.f);
    if (st < ABS_TOL) st = 0.f;
    float xe = 0.f, bhm = 0.f;
    if constexpr (SPIN) {
      xe = fmaxf(vals[GX][k], 0.f);
      if (xe < ABS_TOL) xe = 0.f;
      xe = fminf(xe, 0.999f);
    }
    if constexpr (BH) {
      bhm = fmaxf(vals[GB][k], 0.f);
      if (bhm < ABS_TOL) bhm = 0.f;
    }
    *st_out = st;
    *bhm_out = bhm;
    *dom_out = 1.0 + (double)dx;
    *nf_out = SPIN ? 1.0 - (double)xe : 1.0;
    if constexpr (REC) {
      float nrec = fmaxf(vals[GN][k], 0.f);
      if (nrec < ABS_TOL) nrec = 0.f;
      return (double)nrec / *dom_out;
    }
    return 0.0;
  };
  auto cell = [&](int k) {
    return ((size_t)x * N + y0 + 2 * q + (k & 1)) * N + last_pos<PL>(tq, k >> 1);
  };
  uint32_t Z0 = 0;   // neutral at every radius, yet its closing xH is zero
  bool waited = true;
  int u = 0;
  for (int r = 0; r < bt.nr; ++r) {
    const double pref = bt.fcoll_pref[r];
    const float jaux = bt.J_aux[r], jaux_bh = bt.J_aux_bh[r];
    const bool lastr = FINAL && r == bt.nr - 1;
    X = 0;
    // one (radius, grid) unit; the grid index is a compile-time constant (register arrays)
    auto unit = [&](auto gconst) {
      constexpr int g = decltype(gconst)::value;
      const int b = u % ZB;
      cf* tile = tiles + b * TB;
      if (!mbar_wait(&bars[b], (uint32_t)((u / ZB) & 1), TMA_WAIT_LIMIT)) waited = false;
      line_fft_p<PL, true>(
          tq, tile, s_tw, [&](int p, int) { return ztile_c2r_input<N, Q>(tile, q, p); },
          [&](int p) { return line_addr<N, Q>(p, q); },
          [&](int, cf v, int slot) {
            if constexpr (g < NT) {
              vals[g][2 * slot] = v.x;
              vals[g][2 * slot + 1] = v.y;
            } else {
              // Gamma12 where the cell crossed at this radius, from weighted_sfr and effective_bhar
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                if (!(X & (1u << (2 * slot + h)))) continue;
                const size_t ir = cell(2 * slot + h);
                float f = fmaxf(h ? v.y : v.x, 0.f);
                if (f < ABS_TOL) f = 0.f;
                float G = __fmul_rn(f, g == NT ? bt.G_pref[r] : bt.G_pref_bh[r]);
                if constexpr (BH && g == NT) {
                  vals[1][2 * slot + h] = G;   // stars are used
                } else {
                  if constexpr (BH) G = __fadd_rn(vals[1][2 * slot + h], G);
                  s.Gamma12[ir] = G;
                }
              }
            }
          });
      // every thread is done with tile b (read by the first stage, exchange buffer after that):
      // order those generic accesses before the tensor load that refills it
      fence_proxy_async_smem();
      __syncthreads();
      if (threadIdx.x == 0 && u + ZB < nunits) issue(u + ZB);
      ++u;
      if constexpr (g == NT - 1) {
        // the aliasing clamp (find_HII_bubbles.c:373-422) and the barrier test, both sides
        // times 1 + delta: (f_bh + f_stars) prefactor > nf (1 + rec) with f = grid / dom
        uint32_t M = 0;   // ionised at this radius
#pragma unroll
        for (int k = 0; k < 2 * VL; ++k) {
          float st, bhm;
          double dom, nf;
          const double rec = clamped(k, &st, &bhm, &dom, &nf);
          const double num = BH ? (double)bhm + (double)st : (double)st;
          if (num * pref > nf * (1.0 + rec) * dom) M |= 1u << k;
        }
        if constexpr (REC) X = M & ~I;   // first crossings of the snapshot
        if (FINAL && lastr) {
          // xH = nf - f_coll prefactor where the cell was neutral at every radius, with the sign that
          // says so; that can end below the tolerance too
#pragma unroll
          for (int k = 0; k < 2 * VL; ++k) {
            float xH = 0.f;
            if (!((I | M) >> k & 1u)) {
              float st, bhm;
              double dom, nf;
              clamped(k, &st, &bhm, &dom, &nf);
              const double fcs = (double)st / dom;
              const double fbh = BH ? (double)bhm / dom : 0.0;
              const float w = (float)(nf - (fbh + fcs) * pref);
              xH = w < 0.f ? 0.f : (w > 1.f ? 1.f : w);
              if (xH < REL_TOL) Z0 |= 1u << k;
              xH = -xH;
            }
            s.xH[cell(k)] = xH;
          }
        }
        // new ionizations (find_HII_bubbles.c:531-543) and first crossings (:488-508; Gamma12 follows
        // with the weighted_sfr unit), a small share of the cells
        const uint32_t fresh = (I | M | Z0) & A;
        I |= M;
        if (fresh | X) {
          A &= ~fresh;
#pragma unroll
          for (int k = 0; k < 2 * VL; ++k) {
            const uint32_t bit = 1u << k;
            if (!((fresh | X) & bit)) continue;
            float st, bhm;
            double dom, nf;
            clamped(k, &st, &bhm, &dom, &nf);
            const size_t ir = cell(k);
            if constexpr (REC) {
              if (X & bit) {
                s.r_bubble[ir] = bt.R[r];
                if (c.uvb == 2) {
                  float j = __fmul_rn(st, jaux);
                  if (BH) j = __fadd_rn(j, __fmul_rn(bhm, jaux_bh));
                  s.J21[ir] = j;
                }
              }
            }
            if (fresh & bit) {
              s.z_in[ir] = c.redshift;
              if (c.uvb == 1) {
                float j = st * jaux;
                if (BH) j += bhm * jaux_bh;
                s.J21[ir] = j;
              }
            }
          }
        }
      }
    };
    for_each_index(std::make_integer_sequence<int, NG>{}, unit);
  }
  if (!waited && threadIdx.x % 32 == 0) atomicExch(err, 1u);
  if constexpr (!FINAL) {
    state[0] = (Word)A;
    state[1] = (Word)I;
  }
}

template <int N, bool SPIN, bool BH, bool REC, bool FINAL>
int launch_hii_zr3(rg_context* ctx, const cf* work, int nu, const HiiZUnits& us, cudaStream_t st) {
  using Z = HiiZR<N>;
  constexpr int NG = 2 + SPIN + BH + (REC ? 2 + BH : 0);
  const cf* tw;
  int rc = twiddles_for(ctx, N, &tw);
  if (rc) return rc;
  const HiiBatch& bt = us.u[0].bt;
  // the batch's units as one 3-D float tensor: y (2N floats), x (N), kz of unit u at u NZ + kz
  CUtensorMap map;
  const uint64_t dims[3] = {2ull * N, (uint64_t)N, (uint64_t)Z::NZ * bt.nr * NG * nu};
  const uint64_t strides[2] = {8ull * N, 8ull * N * N};
  const uint32_t box[3] = {4u * Z::Q, 1u, (uint32_t)Z::KZB};
  const int mrc = tma_map_3d(&map, work, dims, strides, box);
  if (mrc != 0) return set_error(ctx, RG_ECUDA, "cuTensorMapEncodeTiled failed (" + std::to_string(mrc) + ")");
  auto kern = k_hii_zr<N, SPIN, BH, REC, FINAL>;
  RG_CUDA_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Z::smem()));
  const double n3 = (double)N * N * N, nzc = (double)Z::NZ * N * N;
  // algorithmic bytes: the Hermitian halves of NG grids per radius, the state (z_at_ionization on
  // the first batch), xH at the end
  prof_begin(ctx, bt.last ? "inv_z_c2r_test_final" : "inv_z_c2r_test", st);
  kern<<<dim3(N / (2 * Z::Q), N, nu), Z::NTH, Z::smem(), st>>>(map, tw, us, ctx->xy_ctrl);
  prof_end(ctx, nu * (bt.nr * NG * 8.0 * nzc + (bt.first || bt.last ? 4.0 * n3 : 0.5 * n3)), st);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  return RG_OK;
}

// nu snapshots (same flags and radii) whose windowed spectra lie one after another in work
template <int N>
int launch_hii_zr(rg_context* ctx, const cf* work, int nu, const HiiZUnits& us, cudaStream_t st) {
  const HiiConst& c = us.u[0].c;
#define RG_ZR(S, B, R)                                                              \
  (us.u[0].bt.last ? launch_hii_zr3<N, S, B, R, true>(ctx, work, nu, us, st) \
                   : launch_hii_zr3<N, S, B, R, false>(ctx, work, nu, us, st))
  if (c.rec)
    return c.spin ? (c.bh ? RG_ZR(true, true, true) : RG_ZR(true, false, true))
                  : (c.bh ? RG_ZR(false, true, true) : RG_ZR(false, false, true));
  return c.spin ? (c.bh ? RG_ZR(true, true, false) : RG_ZR(true, false, false))
                : (c.bh ? RG_ZR(false, true, false) : RG_ZR(false, false, false));
#undef RG_ZR
}

}  // namespace rg
