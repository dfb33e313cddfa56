// Frequency integrals of ComputeTs (ComputeTs.c:761-897) on the device, in FP64: per shell the
// optical-depth-one frequency nu_tau_one (Brent's method over tauX, XRayHeatingFunctions.c:339-424),
// then per (shell, x_e node, kind, band) integrate_over_nu (:742-856), with the adaptive 61-point
// Gauss-Kronrod rule (QUADPACK's QAGE) of the host engine in rg_xray.cpp, which serves the callers
// without a device.
//
// What bounds them: an integral is a chain of rule applications, each 61 evaluations of about a
// thousand dependent FP64 operations; where the interpolated tables jump (their index formula changes at
// 1 keV) the rule halves its interval 20 times to get past it.  So a block takes one integral and
// evaluates the 61 nodes of both halves side by side, each ion's part of the integrand in a group of
// threads of its own, one step a halving.  The integrals of one shell and band share their frequencies:
// the cross sections, spectrum and table positions at the nodes of the first four levels of halvings
// are computed once (k_freq_nodes) for the 42 integrals that read them.
//
// On 8 host threads the integrals took 9 to 10 ms a snapshot (19 ms with both AGN bands), more than the
// rest of a 128^3 snapshot: ComputeTs went from 10.9 to 2.0 ms at 128^3 and from 20.1 to 1.3 ms at 64^3
// with both bands when they moved here, a rule at a time on 64 threads.  In steps of two halves and
// three groups, nu_tau_one and the integrals went from 107 and 652 us (40 shells, on an
// empty device) to 85 and 320, ComputeTs at 128^3 from 1.63 to 1.18 ms.
#include <cfloat>
#include <cstring>
#include <vector>

#include "rg_freq.h"
#include "rg_gk61.h"
#include "rg_xphys.h"

namespace rg {

constexpr int FQ_NT = 64;          // threads of a group: one per rule node (61)
constexpr int FQ_BLOCK = 6 * FQ_NT;   // two intervals, three ions each
constexpr int FQ_LEVELS = 4;       // halvings whose nodes are shared: intervals 0 .. 14 in heap order
constexpr int FQ_SHARED = (1 << FQ_LEVELS) - 1;
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
  int id;   // heap index: the halves of interval i are 2 i + 1 and 2 i + 2
};
__device__ __forceinline__ int fq_child(int id, int right) { return id < FQ_SHARED ? 2 * id + 1 + right : id; }

// A block's integration workspace: the parts of the integrand, the partial sums of each interval's first
// two warps, and the interval list.
struct FqShared {
  double part[2][3][FQ_NT];
  double red[2][2][2][3];   // [phase][interval][warp]
  FqIv iv[FQ_LIMIT];
};

struct FqRule {
  double result, abserr, resabs, resasc;
};

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

// node k of a rule in thread order: lanes 0 .. 29 of the first warp take the nodes left of the centre,
// lane 30 the centre, lanes 0 .. 29 of the second warp those right of it
__device__ __forceinline__ bool fq_node_on(int thread) { return (thread & 31) < 30 || thread == 30; }
__device__ __forceinline__ double fq_node_x(const FreqConst& c, double a, double b, int thread) {
  const double center = 0.5 * (a + b), half = 0.5 * (b - a), d = half * c.X[thread & 31];
  return thread < 32 ? center - d : center + d;
}

// the 61-point rule over n (1 or 2) intervals [iv[h].a, iv[h].b]; f(x, thread of the node, interval id,
// ion) is one ion's part of the integrand.  Every thread of the block gets the same bits.
template <class F>
__device__ void fq_rules(const FreqConst& c, const F& f, const FqIv (&iv)[2], int n, FqShared& sh, FqRule (&out)[2]) {
  const int h = threadIdx.x / (3 * FQ_NT), ion = threadIdx.x / FQ_NT % 3, node = threadIdx.x % FQ_NT, k = node & 31;
  const bool on = h < n && fq_node_on(node);
  const double a = h ? iv[1].a : iv[0].a, b = h ? iv[1].b : iv[0].b;
  sh.part[h][ion][node] = on ? f(fq_node_x(c, a, b, node), node, h ? iv[1].id : iv[0].id, ion) : 0.0;
  __syncthreads();
  const double wk = on ? c.WK[k] : 0.0, wg = on ? c.WG[k] : 0.0;
  const bool adds = ion == 0 && h < n;   // whole warps
  double fx = 0.0;
  if (adds) {
    fx = sh.part[h][0][node] + sh.part[h][1][node] + sh.part[h][2][node];
    double s[3] = {wk * fx, wg * fx, wk * fabs(fx)};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < 3; ++i) s[i] += __shfl_xor_sync(0xffffffffu, s[i], o);
    if (k == 0)
#pragma unroll
      for (int i = 0; i < 3; ++i) sh.red[0][h][node >> 5][i] = s[i];
  }
  __syncthreads();
  if (adds) {
    const double mean = 0.5 * (sh.red[0][h][0][0] + sh.red[0][h][1][0]);
    double d = on ? wk * fabs(fx - mean) : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    if (k == 0) sh.red[1][h][node >> 5][0] = d;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (i >= n) break;
    const double half = 0.5 * (iv[i].b - iv[i].a);
    const double kronrod = sh.red[0][i][0][0] + sh.red[0][i][1][0], gauss = sh.red[0][i][0][1] + sh.red[0][i][1][1];
    out[i].result = kronrod * half;
    out[i].resabs = (sh.red[0][i][0][2] + sh.red[0][i][1][2]) * fabs(half);
    out[i].resasc = (sh.red[1][i][0][0] + sh.red[1][i][1][0]) * fabs(half);
    out[i].abserr = fq_rescale((kronrod - gauss) * half, out[i].resabs, out[i].resasc);
  }
  __syncthreads();   // the sums are read before the next rules write theirs
}

// QAGE; returns 0 on success.  Called by the whole block, the same scalars in every thread.
template <class F>
__device__ int fq_integrate(const FreqConst& c, const F& f, double a, double b, double epsrel, FqShared& sh,
                            double* result) {
  FqIv iv[2] = {FqIv{a, b, 0, 0, 0}, FqIv{a, b, 0, 0, 0}};
  FqRule q[2];
  fq_rules(c, f, iv, 1, sh, q);
  double tolerance = epsrel * fabs(q[0].result);
  const double round_off = 50 * DBL_EPSILON * q[0].resabs;
  *result = q[0].result;
  if (q[0].abserr <= round_off && q[0].abserr > tolerance) return 2;
  if ((q[0].abserr <= tolerance && q[0].abserr != q[0].resasc) || q[0].abserr == 0.0) return 0;
  if (threadIdx.x == 0) sh.iv[0] = FqIv{a, b, q[0].result, q[0].abserr, 0};
  __syncthreads();
  double area = q[0].result, errsum = q[0].abserr;
  int n = 1, type1 = 0, type2 = 0, bad = 0;
  do {
    int im = 0;
    for (int i = 1; i < n; ++i)
      if (sh.iv[i].e > sh.iv[im].e) im = i;
    const FqIv cur = sh.iv[im];
    const double mid = 0.5 * (cur.a + cur.b);
    iv[0] = FqIv{cur.a, mid, 0, 0, fq_child(cur.id, 0)};
    iv[1] = FqIv{mid, cur.b, 0, 0, fq_child(cur.id, 1)};
    fq_rules(c, f, iv, 2, sh, q);   // ends with a barrier: cur is read everywhere
    const double area12 = q[0].result + q[1].result, error12 = q[0].abserr + q[1].abserr;
    errsum += (error12 - cur.e);
    area += area12 - cur.r;
    if (q[0].resasc != q[0].abserr && q[1].resasc != q[1].abserr) {
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
    if (threadIdx.x == 0) {
      sh.iv[im] = FqIv{cur.a, mid, q[0].result, q[0].abserr, iv[0].id};
      sh.iv[n] = FqIv{mid, cur.b, q[1].result, q[1].abserr, iv[1].id};
    }
    __syncthreads();
    ++n;
  } while (n < FQ_LIMIT && !bad && errsum > tolerance);
  double sum = 0;
  for (int i = 0; i < n; ++i) sum += sh.iv[i].r;
  *result = sum;
  __syncthreads();   // the list is read before another integral starts
  if (errsum <= tolerance) return 0;
  return bad ? bad : 1;
}

// tauX(nu, x_e, zp, zpp); 1e10 where the integral fails, as the C does
__device__ double fq_tau(const FreqConst& c, double nu, double zpp, FqShared& sh) {
  const double nu_0 = nu / (1 + c.zp);
  auto f = [&](double z, int, int, int ion) {
    const double opz = (double)(1.0f + (float)z);   // dtdz takes a float redshift
    const double i1 = 1.0 / opz, i3 = i1 * i1 * i1;
    const double dt = c.dtdz_c * (i1 * i1 * sqrt(i1)) / sqrt(c.dtdz_s * i3 + 1);
    const double o = 1 + z;
    const double nu_h = nu_0 * o;
    double fcoll = c.fc0 + (z - c.fcz0) * c.fcslope;
    if (fcoll < 0.0) fcoll = 0.0;
    double ff = fcoll < 1e-20 ? 1 : 1 - (c.ion_eff * fcoll) / (1.0 - c.x_e_ave);
    if (ff < 1e-4) ff = 1e-4;
    double sigma;
    if (ion == 1)
      sigma = c.f_He * (1 - c.x_e_ave) * HeI_ion_crosssec(nu_h);
    else   // the hydrogenic ions
      sigma = (ion == 0 ? c.f_H * (1 - c.x_e_ave) : c.f_He * c.x_e_ave) *
              hydrogenic_crosssec(nu_h, ion == 0 ? NUIONIZATION : HeII_NUIONIZATION, ion == 0 ? SIGMA_HI : 6.3e-18 / 4);
    return SPEED_OF_LIGHT * dt * (c.N_b0 * (o * o * o)) * ff * sigma;
  };
  double r;
  return fq_integrate(c, f, zpp, c.zp, 0.005, sh, &r) ? 1e10 : r;
}

// nu_tau_one: Brent's method on tauX - 1 between the HeI threshold and 1 MeV, to 2 per cent
// (at most 100 iterations), one block per shell
__global__ void __launch_bounds__(FQ_BLOCK) k_freq_tau(const __grid_constant__ FreqConst c, const double* __restrict__ zpps,
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

// limits of a band's integrals for shell r
__device__ __forceinline__ void fq_limits(const FreqConst& c, int band, double zpp, double nu_one, double* lo,
                                          double* hi) {
  const double zf = c.redshifted[band] ? (1. + c.zp) / (1. + zpp) : 1.0;
  *lo = fmax(nu_one, c.lo[band] * zf);
  *hi = c.hi[band] * zf;
}

// the shared nodes of shell blockIdx.x and band blockIdx.y:
// nodes[shell][band][interval][thread of a group][ion]
__global__ void __launch_bounds__(256) k_freq_nodes(const __grid_constant__ FreqConst c,
                                                    const double* __restrict__ zpps, const double* __restrict__ nu_one,
                                                    XNode* __restrict__ nodes) {
  double lo, hi;
  fq_limits(c, blockIdx.y, zpps[blockIdx.x], nu_one[blockIdx.x], &lo, &hi);
  if (!(lo < hi)) return;
  XNode* out = nodes + ((size_t)blockIdx.x * c.nb + blockIdx.y) * FQ_SHARED * FQ_NT * 3;
  const int j = blockIdx.z * 256 + threadIdx.x, ion = j / (FQ_SHARED * FQ_NT), i = j - ion * (FQ_SHARED * FQ_NT);
  if (ion >= 3 || !fq_node_on(i % FQ_NT)) return;
  // the interval's ends by the halvings that lead to it
  double a = lo, b = hi;
  const int id = i / FQ_NT + 1;
  for (int l = 30 - __clz(id); l >= 0; --l) {
    const double mid = 0.5 * (a + b);
    if (id >> l & 1) a = mid;
    else b = mid;
  }
  out[i * 3 + ion] =
      xray_node(ion, c.t.E, c.f_H, c.f_He, c.alpha[blockIdx.y], c.nu_min, fq_node_x(c, a, b, i % FQ_NT));
}

// integrate_over_nu: block (shell, x_e node, 3 band + kind) into out[band][kind][node][shell]
__global__ void __launch_bounds__(FQ_BLOCK)
    k_freq_nu(const __grid_constant__ FreqConst c, const double* __restrict__ zpps, const double* __restrict__ nu_one,
              const XNode* __restrict__ nodes, double* __restrict__ out) {
  __shared__ FqShared sh;
  const int r = blockIdx.x, m = blockIdx.y, band = blockIdx.z / 3, kind = blockIdx.z % 3;
  double lo, hi;
  fq_limits(c, band, zpps[r], nu_one[r], &lo, &hi);
  const double xe = (double)c.t.X[m];
  const XNode* mine = nodes + ((size_t)r * c.nb + band) * FQ_SHARED * FQ_NT * 3;
  double v = 0.0;
  if (lo < hi) {
    auto f = [&](double nu, int node, int id, int ion) {
      const XNode x = id < FQ_SHARED ? mine[(id * FQ_NT + node) * 3 + ion]
                                     : xray_node(ion, c.t.E, c.f_H, c.f_He, c.alpha[band], c.nu_min, nu);
      return xray_part(c.t, kind, ion, xe, nu, x);
    };
    if (fq_integrate(c, f, lo, hi, 0.01, sh, &v))
      v = 0.0;
    else if (kind == 2)
      v *= c.lya;
  }
  if (threadIdx.x == 0) out[((size_t)blockIdx.z * x_int_NXHII + m) * c.nS + r] = v;
}

// the electron tables on the device, uploaded once per table directory
static int freq_tables_on_device(rg_context* ctx, XInt* t) {
  int rc;
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
    // on the stream of the kernels that read them, and there before v goes
    if ((rc = upload(ctx, ctx->freq_xint, v.data(), sizeof(float) * total, ctx->side_stream))) return rc;
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
  // [zpp nS][nu_tau_one nS][tables c.nb 3 14 nS], the same layout on the device and in pinned memory; on
  // the device the shared nodes follow
  const size_t ntab = (size_t)c.nb * 3 * x_int_NXHII * nS, total = 2 * (size_t)nS + ntab;
  const size_t nnode = (size_t)nS * c.nb * FQ_SHARED * FQ_NT * 3;
  static_assert(sizeof(XNode) % sizeof(double) == 0, "nodes behind doubles");
  if ((rc = ensure_device(ctx, &ctx->freq_d, &ctx->freq_d_elems, total + nnode * sizeof(XNode) / sizeof(double))))
    return rc;
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
  XNode* nodes = reinterpret_cast<XNode*>(d + total);
  k_freq_tau<<<nS, FQ_BLOCK, 0, st>>>(c, d, d + nS);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  k_freq_nodes<<<dim3(nS, c.nb, (3 * FQ_SHARED * FQ_NT + 255) / 256), 256, 0, st>>>(c, d, d + nS, nodes);
  RG_CUDA_TRY(ctx, cudaGetLastError());
  k_freq_nu<<<dim3(nS, x_int_NXHII, 3 * c.nb), FQ_BLOCK, 0, st>>>(c, d, d + nS, nodes, d + 2 * nS);
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
