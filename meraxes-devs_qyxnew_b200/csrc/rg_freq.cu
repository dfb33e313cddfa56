// Frequency integrals of ComputeTs (ComputeTs.c:761-897) on the device, in FP64: per shell the
// optical-depth-one frequency nu_tau_one (Brent's method over tauX, XRayHeatingFunctions.c:339-424),
// then per (shell, x_e node, kind, band) integrate_over_nu (:742-856), with the adaptive 61-point
// Gauss-Kronrod rule (QUADPACK's QAGE) of the host engine in rg_xray.cpp, which serves the callers
// without a device.
//
// What bounds it: one integral is a chain of rule applications, each 61 evaluations of about a
// thousand dependent FP64 operations (cross sections, table interpolation), so a block of 64 threads
// evaluates the 61 nodes of a rule side by side and the 1680 integrals of 40 shells (5040 with both
// AGN bands) are 1680 blocks.  On 8 host threads the integrals took 9 to 10 ms a snapshot (19 ms with
// both AGN bands), more than the rest of a 128^3 snapshot: ComputeTs went from 10.9 to 2.0 ms at
// 128^3 and from 20.1 to 1.3 ms at 64^3 with both bands when they moved here.
#include <cfloat>
#include <cstring>
#include <vector>

#include "rg_freq.h"
#include "rg_gk61.h"
#include "rg_xphys.h"

namespace rg {

constexpr int FQ_NT = 64;          // threads of a block: one per rule node (61)
constexpr int FQ_LIMIT = 1000;     // intervals of one adaptive integral
constexpr int FQ_BANDS = 3;        // galaxies, AGN soft, AGN hard

struct FreqConst {
  double X[31], WK[31], WG[31];    // the rule (rg_gk61.h)
  XInt t;
  double N_b0, f_H, f_He;
  double dtdz_c, dtdz_s;           // dt/dz = dtdz_c (1+z)^-2.5 / sqrt(dtdz_s (1+z)^-3 + 1)
  double zp, x_e_ave, ion_eff;
  // collapse fraction interpolated between two snapshots (interpolate_fcoll): f0 + (z - z0) slope
  double fc0, fcz0, fcslope;
  double nu_min;                   // NuXrayThreshold as a frequency
  double lo[FQ_BANDS], hi[FQ_BANDS], alpha[FQ_BANDS];
  int redshifted[FQ_BANDS];        // the band's limits move by (1 + zp) / (1 + zpp) (AGN)
  double lya;                      // prefactor of the Lyman-alpha integral
  int nS, nb;
};

struct FqIv {
  double a, b, r, e;
};

// A block's integration workspace: partial sums of its two warps and the interval list.
struct FqShared {
  double red[2][2][3];
  FqIv iv[FQ_LIMIT];
};

// Sum of K values over the block; every thread gets the same bits.  `phase` alternates the buffer.
template <int K>
__device__ __forceinline__ void fq_sum(double (&v)[K], FqShared& sh, int phase) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int k = 0; k < K; ++k) sh.red[phase][threadIdx.x >> 5][k] = v[k];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; ++k) v[k] = sh.red[phase][0][k] + sh.red[phase][1][k];
}

__device__ __forceinline__ double fq_rescale(double err, double result_abs, double result_asc) {
  err = fabs(err);
  if (result_asc != 0 && err != 0) {
    const double s = 200 * err / result_asc, scale = s * sqrt(s);
    err = scale < 1 ? result_asc * scale : result_asc;
  }
  if (result_abs > DBL_MIN / (50 * DBL_EPSILON)) {
    const double min_err = 50 * DBL_EPSILON * result_abs;
    if (min_err > err) err = min_err;
  }
  return err;
}

// the 61-point rule over [a, b]: thread k < 30 of each warp takes node k on its side of the centre,
// thread 30 of the first warp the centre
template <class F>
__device__ void fq_rule(const FreqConst& c, const F& f, double a, double b, FqShared& sh, double* result,
                        double* abserr, double* resabs, double* resasc) {
  const int k = threadIdx.x & 31, side = threadIdx.x >> 5;
  const double center = 0.5 * (a + b), half = 0.5 * (b - a);
  const bool on = k < 30 || (k == 30 && side == 0);
  double fx = 0, wk = 0, wg = 0;
  if (on) {
    const double d = half * c.X[k];
    fx = f(side ? center + d : center - d);
    wk = c.WK[k];
    wg = c.WG[k];
  }
  double s[3] = {wk * fx, wg * fx, wk * fabs(fx)};
  fq_sum<3>(s, sh, 0);
  const double mean = 0.5 * s[0];
  double asc[1] = {on ? wk * fabs(fx - mean) : 0.0};
  fq_sum<1>(asc, sh, 1);
  *result = s[0] * half;
  *resabs = s[2] * fabs(half);
  *resasc = asc[0] * fabs(half);
  *abserr = fq_rescale((s[0] - s[1]) * half, *resabs, *resasc);
}

// QAGE; returns 0 on success.  Called by the whole block, the same scalars in every thread.
template <class F>
__device__ int fq_integrate(const FreqConst& c, const F& f, double a, double b, double epsrel, FqShared& sh,
                            double* result) {
  double r0, e0, ra0, rc0;
  fq_rule(c, f, a, b, sh, &r0, &e0, &ra0, &rc0);
  double tolerance = epsrel * fabs(r0);
  const double round_off = 50 * DBL_EPSILON * ra0;
  *result = r0;
  if (e0 <= round_off && e0 > tolerance) return 2;
  if ((e0 <= tolerance && e0 != rc0) || e0 == 0.0) return 0;
  __syncthreads();   // readers of an earlier integral's list are done
  if (threadIdx.x == 0) sh.iv[0] = FqIv{a, b, r0, e0};
  __syncthreads();
  double area = r0, errsum = e0;
  int n = 1, type1 = 0, type2 = 0, bad = 0;
  do {
    int im = 0;
    for (int i = 1; i < n; ++i)
      if (sh.iv[i].e > sh.iv[im].e) im = i;
    const FqIv cur = sh.iv[im];
    const double mid = 0.5 * (cur.a + cur.b);
    double a1, e1, ab1, as1, a2, e2, ab2, as2;
    fq_rule(c, f, cur.a, mid, sh, &a1, &e1, &ab1, &as1);
    fq_rule(c, f, mid, cur.b, sh, &a2, &e2, &ab2, &as2);
    const double area12 = a1 + a2, error12 = e1 + e2;
    errsum += (error12 - cur.e);
    area += area12 - cur.r;
    if (as1 != e1 && as2 != e2) {
      const double delta = cur.r - area12;
      if (fabs(delta) <= 1.0e-5 * fabs(area12) && error12 >= 0.99 * cur.e) type1++;
      if (n >= 10 && error12 > cur.e) type2++;
    }
    tolerance = epsrel * fabs(area);
    if (errsum > tolerance) {
      if (type1 >= 6 || type2 >= 20) bad = 2;
      const double tmp = (1 + 100 * DBL_EPSILON) * (fabs(mid) + 1000 * DBL_MIN);
      if (fabs(cur.a) <= tmp && fabs(cur.b) <= tmp) bad = 3;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      sh.iv[im] = FqIv{cur.a, mid, a1, e1};
      sh.iv[n] = FqIv{mid, cur.b, a2, e2};
    }
    __syncthreads();
    ++n;
  } while (n < FQ_LIMIT && !bad && errsum > tolerance);
  double sum = 0;
  for (int i = 0; i < n; ++i) sum += sh.iv[i].r;
  *result = sum;
  if (errsum <= tolerance) return 0;
  return bad ? bad : 1;
}

// tauX(nu, x_e, zp, zpp); 1e10 where the integral fails, as the C does
__device__ double fq_tau(const FreqConst& c, double nu, double zpp, FqShared& sh) {
  const double nu_0 = nu / (1 + c.zp);
  auto f = [&](double z) {
    const double opz = (double)(1.0f + (float)z);   // dtdz takes a float redshift
    const double i1 = 1.0 / opz, i3 = i1 * i1 * i1;
    const double dt = c.dtdz_c * (i1 * i1 * sqrt(i1)) / sqrt(c.dtdz_s * i3 + 1);
    const double o = 1 + z;
    const double nu_h = nu_0 * o;
    double fcoll = c.fc0 + (z - c.fcz0) * c.fcslope;
    if (fcoll < 0.0) fcoll = 0.0;
    double ff = fcoll < 1e-20 ? 1 : 1 - (c.ion_eff * fcoll) / (1.0 - c.x_e_ave);
    if (ff < 1e-4) ff = 1e-4;
    const double sigma = c.f_H * (1 - c.x_e_ave) * HI_ion_crosssec(nu_h) +
                         c.f_He * (1 - c.x_e_ave) * HeI_ion_crosssec(nu_h) + c.f_He * c.x_e_ave * HeII_ion_crosssec(nu_h);
    return SPEED_OF_LIGHT * dt * (c.N_b0 * (o * o * o)) * ff * sigma;
  };
  double r;
  return fq_integrate(c, f, zpp, c.zp, 0.005, sh, &r) ? 1e10 : r;
}

// nu_tau_one: Brent's method on tauX - 1 between the HeI threshold and 1 MeV, to 2 per cent
// (at most 100 iterations), one block per shell
__global__ void __launch_bounds__(FQ_NT) k_freq_tau(const __grid_constant__ FreqConst c, const double* __restrict__ zpps,
                                                    double* __restrict__ nu_one) {
  __shared__ FqShared sh;
  const double zpp = zpps[blockIdx.x];
  auto fn = [&](double nu) { return fq_tau(c, nu, zpp, sh) - 1; };
  double root;
  if (c.x_e_ave > 0.9999) {
    root = -1.0;
  } else {
    double a = HeI_NUIONIZATION, b = 1e6 * NU_over_EV;
    double fa = fn(a), fb;
    if (fa < 0) {
      root = a;
    } else if ((fb = fn(b)) > 0.0 && fa > 0.0) {
      root = b;   // no sign change
    } else {
      double e1 = b, fc = fb, d = b - a, e = b - a;   // e1: the contrapoint
      root = b;
      double lo = a, hi = b;
      for (int it = 0; it < 100; ++it) {
        bool two = false;
        if ((fb < 0 && fc < 0) || (fb > 0 && fc > 0)) {
          two = true;
          e1 = a;
          fc = fa;
          d = b - a;
          e = b - a;
        }
        if (fabs(fc) < fabs(fb)) {
          two = true;
          a = b;
          b = e1;
          e1 = a;
          fa = fb;
          fb = fc;
          fc = fa;
        }
        const double tol = 0.5 * DBL_EPSILON * fabs(b);
        const double m = 0.5 * (e1 - b);
        if (fb == 0) {
          root = lo = hi = b;
        } else if (fabs(m) <= tol) {
          root = b;
          lo = b < e1 ? b : e1;
          hi = b < e1 ? e1 : b;
        } else {
          if (fabs(e) < tol || fabs(fa) <= fabs(fb)) {
            d = m;
            e = m;
          } else {
            double p, q;
            const double s = fb / fa;
            if (two) {
              p = 2 * m * s;
              q = 1 - s;
            } else {
              q = fa / fc;
              const double r = fb / fc;
              p = s * (2 * m * q * (q - r) - (b - a) * (r - 1));
              q = (q - 1) * (r - 1) * (s - 1);
            }
            if (p > 0)
              q = -q;
            else
              p = -p;
            if (2 * p < fmin(3 * m * q - fabs(tol * q), fabs(e * q))) {
              e = d;
              d = p / q;
            } else {
              d = m;
              e = m;
            }
          }
          a = b;
          fa = fb;
          if (fabs(d) > tol)
            b += d;
          else
            b += (m > 0 ? +tol : -tol);
          fb = fn(b);
          root = b;
          if ((fb < 0 && fc < 0) || (fb > 0 && fc > 0)) e1 = a;
          lo = b < e1 ? b : e1;
          hi = b < e1 ? e1 : b;
        }
        const double least = ((lo > 0 && hi > 0) || (lo < 0 && hi < 0)) ? fmin(fabs(lo), fabs(hi)) : 0;
        if (fabs(hi - lo) < 0.02 * least) break;
      }
    }
  }
  if (threadIdx.x == 0) nu_one[blockIdx.x] = root;
}

// integrate_over_nu: block (shell, x_e node, 3 band + kind) into out[band][kind][node][shell]
__global__ void __launch_bounds__(FQ_NT)
    k_freq_nu(const __grid_constant__ FreqConst c, const double* __restrict__ zpps, const double* __restrict__ nu_one,
              double* __restrict__ out) {
  __shared__ FqShared sh;
  const int r = blockIdx.x, m = blockIdx.y, band = blockIdx.z / 3, kind = blockIdx.z % 3;
  const double zf = c.redshifted[band] ? (1. + c.zp) / (1. + zpps[r]) : 1.0;
  const double lo = fmax(nu_one[r], c.lo[band] * zf), hi = c.hi[band] * zf;
  const double xe = (double)c.t.X[m];
  double v = 0.0;
  if (lo < hi) {
    auto f = [&](double nu) { return xray_integrand(c.t, c.f_H, c.f_He, kind, xe, c.alpha[band], c.nu_min, nu); };
    if (fq_integrate(c, f, lo, hi, 0.01, sh, &v))
      v = 0.0;
    else if (kind == 2)
      v *= c.lya;
  }
  if (threadIdx.x == 0) out[((size_t)blockIdx.z * x_int_NXHII + m) * c.nS + r] = v;
}

// the electron tables on the device, uploaded once per table directory
static int freq_tables_on_device(rg_context* ctx, XInt* t) {
  const Tables& h = ctx->tables;
  const size_t per = (size_t)x_int_NXHII * x_int_NENERGY, total = x_int_NENERGY + x_int_NXHII + 5 * per;
  if (!ctx->freq_xint || ctx->freq_dir != h.dir) {
    if (!ctx->freq_xint && cudaMalloc((void**)&ctx->freq_xint, sizeof(float) * total) != cudaSuccess) {
      ctx->freq_xint = nullptr;
      return set_error(ctx, RG_ENOMEM, "cudaMalloc of the electron tables failed");
    }
    std::vector<float> v;
    v.reserve(total);
    for (const std::vector<float>* a :
         {&h.x_int_Energy, &h.x_int_XHII, &h.fheat, &h.n_Lya, &h.nion_HI, &h.nion_HeI, &h.nion_HeII})
      v.insert(v.end(), a->begin(), a->end());
    ctx->freq_dir.clear();
    RG_CUDA_TRY(ctx, cudaMemcpy(ctx->freq_xint, v.data(), sizeof(float) * total, cudaMemcpyHostToDevice));
    ctx->freq_dir = h.dir;
  }
  const float* b = ctx->freq_xint;
  t->E = b;
  t->X = b + x_int_NENERGY;
  const float* tab = t->X + x_int_NXHII;
  t->fheat = tab;
  t->n_Lya = tab + per;
  t->nion_HI = tab + 2 * per;
  t->nion_HeI = tab + 3 * per;
  t->nion_HeII = tab + 4 * per;
  return RG_OK;
}

// bands of a snapshot: the galaxies', then the AGN bands Flag_IncludeAGNXray uses (0 soft, 1 hard)
static int freq_bands(const rg_params* p, int* agn) {
  const int f = p->Flag_IncludeAGNXray;
  int n = 0;
  if (f == 1 || f == 3) agn[n++] = 0;
  if (f == 1 || f == 2) agn[n++] = 1;
  return n;
}

int ts_freq_start(rg_context* ctx, const rg_params* p, const TsShells& sh, double zp, double x_e_ave,
                  double collapse_fraction, const double* ZZ, const double* stored_fcoll, int snapshot) {
  int rc;
  FreqConst c;
  std::memset(&c, 0, sizeof(c));
  std::memcpy(c.X, GK61_X, sizeof(c.X));
  std::memcpy(c.WK, GK61_WK, sizeof(c.WK));
  std::memcpy(c.WG, GK61_WG, sizeof(c.WG));
  // nothing of an earlier call is in flight on the side stream (an error may have left it there)
  RG_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->side_stream));
  if ((rc = freq_tables_on_device(ctx, &c.t))) return rc;
  const Cosmo cm(p);
  c.N_b0 = cm.N_b0;
  c.f_H = cm.f_H;
  c.f_He = cm.f_He;
  // Cosmo::dtdz in one fraction: c (x' (1 + x / s)) / (x + s) = c x' / s with s = sqrt(x^2 + 1)
  const double lm = p->OmegaLambda / p->OmegaM;
  c.dtdz_c = 2 * std::sqrt(1 + 1 / lm) / (3.0 * HUBBLE * p->Hubble_h) * std::sqrt(lm) * (-3.0 / 2.0);
  c.dtdz_s = lm;
  c.zp = zp;
  c.x_e_ave = x_e_ave;
  c.ion_eff = p->ReionEfficiency;
  if (snapshot == 0) {
    c.fc0 = collapse_fraction;
  } else {
    c.fc0 = stored_fcoll[snapshot - 1];
    c.fcz0 = ZZ[snapshot - 1];
    c.fcslope = (collapse_fraction - stored_fcoll[snapshot - 1]) / (ZZ[snapshot] - ZZ[snapshot - 1]);
  }
  c.nu_min = p->NuXrayThreshold * NU_over_EV;
  c.lo[0] = c.nu_min;
  c.hi[0] = p->NuXrayMax * NU_over_EV;
  c.alpha[0] = p->SpecIndexXrayGal;
  int agn[2];
  const int na = freq_bands(p, agn);
  for (int j = 0; j < na; ++j) {
    const bool hard = agn[j] == 1;
    c.lo[1 + j] = (hard ? p->NuXraySoftCut : p->NuXrayThreshold) * NU_over_EV;
    c.hi[1 + j] = (hard ? p->NuXrayMax : p->NuXraySoftCut) * NU_over_EV;
    c.alpha[1 + j] = hard ? p->SpecIndexXrayAGNHard : p->SpecIndexXrayAGNSoft;
    c.redshifted[1 + j] = 1;
  }
  c.lya = SPEED_OF_LIGHT / (4 * M_PI) / NU_LA / cm.hubble((float)zp);
  const int nS = sh.nS;
  c.nS = nS;
  c.nb = 1 + na;
  // [zpp nS][nu_tau_one nS][tables c.nb 3 14 nS], the same layout on the device and in pinned memory
  const size_t ntab = (size_t)c.nb * 3 * x_int_NXHII * nS, total = 2 * (size_t)nS + ntab;
  if ((rc = ensure_device(ctx, &ctx->freq_d, &ctx->freq_d_elems, total))) return rc;
  if (ctx->freq_h_elems < total) {
    if (ctx->freq_h) cudaFreeHost(ctx->freq_h);
    ctx->freq_h = nullptr;
    ctx->freq_h_elems = 0;
    if (cudaMallocHost((void**)&ctx->freq_h, sizeof(double) * total) != cudaSuccess)
      return set_error(ctx, RG_ENOMEM, "pinned frequency tables");
    ctx->freq_h_elems = total;
  }
  for (int r = 0; r < nS; ++r)
    ctx->freq_h[r] = (sh.zpp_edge[r] + (r == 0 ? zp : sh.zpp_edge[r - 1])) * 0.5;
  cudaStream_t st = ctx->side_stream;
  double* d = ctx->freq_d;
  RG_CUDA_TRY(ctx, cudaMemcpyAsync(d, ctx->freq_h, sizeof(double) * nS, cudaMemcpyHostToDevice, st));
  k_freq_tau<<<nS, FQ_NT, 0, st>>>(c, d, d + nS);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  k_freq_nu<<<dim3(nS, x_int_NXHII, 3 * c.nb), FQ_NT, 0, st>>>(c, d, d + nS, d + 2 * nS);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  RG_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->freq_h + nS, d + nS, sizeof(double) * (total - nS), cudaMemcpyDeviceToHost, st));
  return RG_OK;
}

int ts_freq_finish(rg_context* ctx, const rg_params* p, const TsShells& sh, double zp, TsTables* out) {
  ts_sum_lyn(ctx->tables, p, sh, zp, &out->sum_lyn);   // while the device integrates
  RG_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->side_stream));
  const int nS = sh.nS;
  const size_t per = (size_t)x_int_NXHII * nS;
  const double* t = ctx->freq_h + 2 * nS;
  out->heat.assign(t, t + per);
  out->ion.assign(t + per, t + 2 * per);
  out->lya.assign(t + 2 * per, t + 3 * per);
  int agn[2];
  const int na = freq_bands(p, agn);
  for (int j = 0; j < na; ++j)
    for (int k = 0; k < 3; ++k) {
      const double* a = t + (size_t)(3 * (1 + j) + k) * per;
      out->agn[agn[j]][k].assign(a, a + per);
    }
  return RG_OK;
}

}  // namespace rg
