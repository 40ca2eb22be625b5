// coef.h -- Metropolis coefficients from the material parameters and T.
//
// One function, compiled for the host runtime (g++ -ffp-contract=off) and for
// the device swap kernel (nvcc -fmad=false), so that a replica whose
// temperature changes on the device gets bit-for-bit the coefficients the host
// would have computed.
#pragma once
#include "mmc_internal.h"

namespace mmc {

// Temperature-independent inputs of McCoef (SI).
struct McParams {
  double aex, dind, ku1, ms;
  double b[3];
  double u[3];     // normalised anisotropy axis
  double d[3];
  double v;        // dx dy dz
  double mu0;
  double k0[6];    // self tensor (0 when demag is off)
  int demag;
  uint32_t key0, key1;
};

#if defined(__CUDACC__)
#define MMC_COEF_HD __host__ __device__
#else
#define MMC_COEF_HD
#endif

// The FP32 filter's coefficients from the FP64 ones.  |F_a| of a trial is at
// most (2 sum wex + 2 sum |wdm| + 3 k0h (1 + 1) + 2 can (1 + 1)) max(1, |m|) +
// |cz| + cd |h|, components at most max(1, |m|) and |h|.
MMC_COEF_HD inline McFilter mc_filter_from(const McCoef<double>& k) {
  McFilter f;
  double g = 0, gz = 0, kmax = 0, cmax = 0;
  for (int a = 0; a < 3; ++a) {
    f.wex[a] = (float)k.wex[a];
    f.u[a] = (float)k.u[a];
    f.cz[a] = (float)k.cz[a];
    (a < 2 ? g : gz) += 2.0 * (k.wex[a] < 0 ? -k.wex[a] : k.wex[a]);
    const double z = k.cz[a] < 0 ? -k.cz[a] : k.cz[a];
    if (!(z <= cmax)) cmax = z;
  }
  for (int a = 0; a < 2; ++a) {
    f.wdm[a] = (float)k.wdm[a];
    g += 2.0 * (k.wdm[a] < 0 ? -k.wdm[a] : k.wdm[a]);
  }
  for (int q = 0; q < 6; ++q) {
    f.k0h[q] = (float)k.k0h[q];
    const double z = k.k0h[q] < 0 ? -k.k0h[q] : k.k0h[q];
    if (!(z <= kmax)) kmax = z;
  }
  f.can = (float)k.can;
  f.cd = (float)k.cd;
  g += 6.0 * kmax + 4.0 * (k.can < 0 ? -k.can : k.can);
  f.gm = (float)(1.001 * g);
  f.gz = (float)(1.001 * gz);
  f.gc = (float)(1.001 * cmax);
  return f;
}

template <typename T>
MMC_COEF_HD inline McCoef<T> mc_coef_from(const McParams& p, double T_K) {
  const double kB = 1.3806488e-23;  // src/constant.h:22
  const double kT = kB * T_K;
  McCoef<T> k;
  for (int a = 0; a < 3; ++a) k.wex[a] = (T)(2.0 * p.aex * p.v / (p.d[a] * p.d[a] * kT));
  k.wdm[0] = (T)(p.dind * p.v / (p.d[0] * kT));
  k.wdm[1] = (T)(p.dind * p.v / (p.d[1] * kT));
  k.can = (T)(p.ku1 * p.v / kT);
  for (int a = 0; a < 3; ++a) k.u[a] = (T)p.u[a];
  k.cz[0] = (T)(p.ms * p.v * p.b[0] / kT);
  k.cz[1] = (T)(p.ms * p.v * p.b[1] / kT);
  k.cz[2] = (T)(p.ms * p.v * p.b[2] / kT);
  k.cd = (T)(p.demag ? p.mu0 * p.ms * p.ms * p.v / kT : 0.0);
  for (int q = 0; q < 6; ++q) k.k0[q] = (T)(p.demag ? p.k0[q] : 0.0);
  for (int q = 0; q < 6; ++q) k.k0h[q] = (T)(p.demag ? 0.5 * (p.mu0 * p.ms * p.ms * p.v / kT) * p.k0[q] : 0.0);
  k.key0 = p.key0;
  k.key1 = p.key1;
  if constexpr (sizeof(T) == 8) k.f = mc_filter_from(k);
  return k;
}

}  // namespace mmc
