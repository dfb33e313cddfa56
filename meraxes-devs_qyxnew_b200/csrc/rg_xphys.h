// The integrands of the X-ray frequency integrals, for the host engine (rg_xray.cpp) and the device
// kernels (rg_freq.cu): photo-ionisation cross sections (XRayHeatingFunctions.c:471-516), the
// electron interpolation tables (:970-1276) and the heating / ionisation / Lyman-alpha integrands
// of integrate_over_nu (:742-856).
#pragma once

#include <math.h>

#include "rg_internal.h"

#ifdef __CUDACC__
#define RG_HD __host__ __device__
#else
#define RG_HD
#endif

namespace rg {

RG_HD inline double HeI_ion_crosssec(double nu) {
  if (nu < HeI_NUIONIZATION) return 0;
  const double x = nu / NU_over_EV / 13.61 - 0.4434;
  const double y = sqrt(x * x + 2.136 * 2.136);
  return 9.492e-16 * ((x - 1) * (x - 1) + 2.039 * 2.039) * pow(y, (0.5 * 3.188 - 5.5)) *
         pow(1.0 + sqrt(y / 1.469), -3.188);
}

// hydrogenic ions: sigma0 / Z^2 (nu0 / nu)^4 exp(4 - 4 atan(e) / e) / (1 - exp(-2 pi / e))
RG_HD inline double hydrogenic_crosssec(double nu, double nu0, double sigma) {
  if (nu < nu0) return 0;
  if (nu == nu0) nu += TINY;
  const double epsilon = sqrt(nu / nu0 - 1);
  const double r = nu0 / nu, r2 = r * r;
  return sigma * (r2 * r2) * exp(4 - (4 * atan(epsilon) / epsilon)) / (1 - exp(-2 * M_PI / epsilon));
}
RG_HD inline double HeII_ion_crosssec(double nu) { return hydrogenic_crosssec(nu, HeII_NUIONIZATION, 6.3e-18 / 4); }
RG_HD inline double HI_ion_crosssec(double nu) { return hydrogenic_crosssec(nu, NUIONIZATION, SIGMA_HI); }

// The electron tables: energies E[258], x_HII nodes X[14], and per table [14][258] values.
struct XInt {
  const float *E, *X;
  const float *fheat, *n_Lya, *nion_HI, *nion_HeI, *nion_HeII;
};

RG_HD inline int locate_energy_index(float En) {
  if (En < 1008.88f) return (int)(log((double)En / 10.0) / 1.98026273e-2);
  return 232 + (int)(log((double)En / 1008.88) / 9.53101798e-2);
}

// the last node not above x (x is at least X[0])
RG_HD inline int locate_xHII_index(const float* X, float x) {
  int m = x_int_NXHII - 1;
  while (m > 0 && x < X[m]) m--;
  return m;
}

RG_HD inline double xray_ion(int i) { return i == 0 ? NUIONIZATION : i == 1 ? HeI_NUIONIZATION : HeII_NUIONIZATION; }

// What the integrands of one frequency share for an ion (0 HI, 1 HeI, 2 HeII), whatever the x_e and the
// kind: the cross section times its number fraction and the spectrum (nu / nu0)^(-alpha - 1), the
// electron energy within the tables and the energy interval it lies in (-1: below the tables).
struct XNode {
  double g;
  float en;
  int lo;
};

// nu0: the threshold frequency the spectrum is normalised at
RG_HD inline XNode xray_node(int ion, const float* E, double f_H, double f_He, double alpha, double nu0, double nu) {
  XNode x;
  const double sigma = ion == 1 ? HeI_ion_crosssec(nu)
                                : hydrogenic_crosssec(nu, ion == 0 ? NUIONIZATION : HeII_NUIONIZATION,
                                                      ion == 0 ? SIGMA_HI : 6.3e-18 / 4);
  x.g = (ion == 0 ? f_H : f_He) * sigma * pow(nu / nu0, -alpha - 1);
  x.en = (float)((nu - xray_ion(ion)) / NU_over_EV);
  if ((double)x.en > 0.999 * (double)E[x_int_NENERGY - 1]) x.en = (float)((double)E[x_int_NENERGY - 1] * 0.999);
  x.lo = x.en < E[0] ? -1 : locate_energy_index(x.en);
  return x;
}

// bilinear interpolation of one table at (energy en in interval n_low, x_e xf), float arithmetic in the
// order of the C
RG_HD inline float interp_x_int(const XInt& t, const float* tab, float en, int n_low, float xf, float below) {
  const float *E = t.E, *X = t.X;
  if (n_low < 0) return below;
  if ((double)xf > (double)X[x_int_NXHII - 1] * 0.999) {
    xf = (float)((double)X[x_int_NXHII - 1] * 0.999);
  } else if (xf < X[0]) {
    xf = (float)(1.001 * (double)X[0]);
  }
  const int n_high = n_low + 1;
  const int m_low = locate_xHII_index(X, xf), m_high = m_low + 1;
  const float* lo = tab + m_low * x_int_NENERGY;
  const float* hi = tab + m_high * x_int_NENERGY;
  float elow = ((lo[n_high] - lo[n_low]) / (E[n_high] - E[n_low]));
  elow *= (en - E[n_low]);
  elow += lo[n_low];
  float ehigh = ((hi[n_high] - hi[n_low]) / (E[n_high] - E[n_low]));
  ehigh *= (en - E[n_low]);
  ehigh += hi[n_low];
  float r = (ehigh - elow) / (X[m_high] - X[m_low]);
  r *= (xf - X[m_low]);
  r += elow;
  return r;
}

// an ion's part of the integrand of integrate_over_nu at frequency nu: kind 0 heating, 1 ionisation,
// 2 Lyman-alpha
RG_HD inline double xray_part(const XInt& t, int kind, int ion, double x_e, double nu, const XNode& x) {
  const float xf = (float)x_e;
  const double g = x.g * (ion < 2 ? 1 - x_e : x_e);
  if (kind == 0) return interp_x_int(t, t.fheat, x.en, x.lo, xf, 1.0f) * PLANCK * (nu - xray_ion(ion)) * g;
  if (kind == 1)
    return (interp_x_int(t, t.nion_HI, x.en, x.lo, xf, 0.0f) + interp_x_int(t, t.nion_HeI, x.en, x.lo, xf, 0.0f) +
            interp_x_int(t, t.nion_HeII, x.en, x.lo, xf, 0.0f) + 1) *
           g;
  return interp_x_int(t, t.n_Lya, x.en, x.lo, xf, 0.0f) * g;
}

}  // namespace rg
