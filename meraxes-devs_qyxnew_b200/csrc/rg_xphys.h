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

// bilinear interpolation of one table, float arithmetic in the order of the C
RG_HD inline float interp_x_int(const XInt& t, const float* tab, float En, float xHII_call, float below) {
  const float *E = t.E, *X = t.X;
  if ((double)En > 0.999 * (double)E[x_int_NENERGY - 1]) {
    En = (float)((double)E[x_int_NENERGY - 1] * 0.999);
  } else if (En < E[0]) {
    return below;
  }
  if ((double)xHII_call > (double)X[x_int_NXHII - 1] * 0.999) {
    xHII_call = (float)((double)X[x_int_NXHII - 1] * 0.999);
  } else if (xHII_call < X[0]) {
    xHII_call = (float)(1.001 * (double)X[0]);
  }
  const int n_low = locate_energy_index(En), n_high = n_low + 1;
  const int m_low = locate_xHII_index(X, xHII_call), m_high = m_low + 1;
  const float* lo = tab + m_low * x_int_NENERGY;
  const float* hi = tab + m_high * x_int_NENERGY;
  float elow = ((lo[n_high] - lo[n_low]) / (E[n_high] - E[n_low]));
  elow *= (En - E[n_low]);
  elow += lo[n_low];
  float ehigh = ((hi[n_high] - hi[n_low]) / (E[n_high] - E[n_low]));
  ehigh *= (En - E[n_low]);
  ehigh += hi[n_low];
  float r = (ehigh - elow) / (X[m_high] - X[m_low]);
  r *= (xHII_call - X[m_low]);
  r += elow;
  return r;
}

// integrand of integrate_over_nu: kind 0 heating, 1 ionisation, 2 Lyman-alpha; nu0 the threshold
// frequency the spectrum nu^-alpha is normalised at
RG_HD inline double xray_integrand(const XInt& t, double f_H, double f_He, int kind, double x_e, double alpha,
                                   double nu0, double nu) {
  const float xf = (float)x_e;
  const double ion[3] = {NUIONIZATION, HeI_NUIONIZATION, HeII_NUIONIZATION};
  const double sig[3] = {f_H * (1 - x_e) * HI_ion_crosssec(nu), f_He * (1 - x_e) * HeI_ion_crosssec(nu),
                         f_He * x_e * HeII_ion_crosssec(nu)};
  double s = 0;
  for (int i = 0; i < 3; ++i) {
    const float en = (float)((nu - ion[i]) / NU_over_EV);
    if (kind == 0)
      s += interp_x_int(t, t.fheat, en, xf, 1.0f) * PLANCK * (nu - ion[i]) * sig[i];
    else if (kind == 1)
      s += (interp_x_int(t, t.nion_HI, en, xf, 0.0f) + interp_x_int(t, t.nion_HeI, en, xf, 0.0f) +
            interp_x_int(t, t.nion_HeII, en, xf, 0.0f) + 1) *
           sig[i];
    else
      s += interp_x_int(t, t.n_Lya, en, xf, 0.0f) * sig[i];
  }
  return s * pow(nu / nu0, -alpha - 1);
}

}  // namespace rg
