// Device math shared by the setup and operator kernels.
//
// Expansions use the real form of pi-BEM's complex solid-harmonic coefficients
// (include/multipole_expansion.h:102-105): K = (p+1)^2 reals per expansion,
// for each degree n the real part of m = 0 followed by (re, im) of m = 1..n.
// Multipole coefficients are scaled by the box side h (M^_n = M_n / h^n) and
// local coefficients by h^(n+1) (L^_n = L_n h^(n+1)).
#pragma once

#include <cuda_runtime.h>

#include <cmath>

namespace pibem
{
  // (n, m, part) of real index k.
  __host__ __device__ inline void real_index(int k, int &n, int &m, int &part)
  {
    n = 0;
    while ((n + 1) * (n + 1) <= k)
      ++n;
    int r = k - n * n;
    if (r == 0)
      {
        m    = 0;
        part = 0;
      }
    else
      {
        m    = (r + 1) / 2;
        part = (r + 1) % 2; // r odd -> re, even -> im
      }
  }

  // Normalised associated Legendre functions P~_n^m(x) = sqrt((n-m)!/(n+m)!) P_n^m(x),
  // Condon-Shortley phase (the normalisation of source/ass_leg_function.cc), by the
  // three-term recurrence in n; s = sqrt(1-x^2).
  // Coefficients of the normalised Legendre recurrences for n, m <= 20:
  //   P~_m^m     = -cmm[m] s P~_{m-1}^{m-1},       cmm[m] = sqrt((2m-1)/(2m))
  //   P~_{m+1}^m = cm1[m] x P~_m^m,                cm1[m] = sqrt(2m+1)
  //   P~_n^m     = ra[n][m] x P~_{n-1}^m - rb[n][m] P~_{n-2}^m,
  //                ra = (2n-1)/sqrt(n^2-m^2), rb = sqrt((n-1)^2-m^2)/sqrt(n^2-m^2)
  struct LegendreTables
  {
    double cmm[21], cm1[21], ra[21][21], rb[21][21];
    float  fcmm[21], fcm1[21], fra[21][21], frb[21][21];
    float2 ffcmm[21], ffcm1[21], ffra[21][21], ffrb[21][21]; // (hi, lo) pairs
  };
  // One copy per translation unit that evaluates expansions; filled by
  // fill_legendre_tables() + cudaMemcpyToSymbol from that unit.
  static __constant__ LegendreTables c_leg;

  inline void fill_legendre_tables(LegendreTables &t)
  {
    auto pair = [](double v) {
      const float hi = float(v);
      return make_float2(hi, float(v - double(hi)));
    };
    for (int m = 0; m <= 20; ++m)
      {
        t.cmm[m] = m > 0 ? std::sqrt((2.0 * m - 1.0) / (2.0 * m)) : 0.0;
        t.cm1[m] = std::sqrt(2.0 * m + 1.0);
        for (int n = 0; n <= 20; ++n)
          {
            bool ok    = n >= m + 2;
            t.ra[n][m] = ok ? (2.0 * n - 1.0) / std::sqrt(double(n * n - m * m)) : 0.0;
            t.rb[n][m] = ok ? std::sqrt(double((n - 1) * (n - 1) - m * m)) / std::sqrt(double(n * n - m * m)) : 0.0;
            t.fra[n][m] = float(t.ra[n][m]);
            t.frb[n][m] = float(t.rb[n][m]);
            t.ffra[n][m] = pair(t.ra[n][m]);
            t.ffrb[n][m] = pair(t.rb[n][m]);
          }
        t.fcmm[m] = float(t.cmm[m]);
        t.fcm1[m] = float(t.cm1[m]);
        t.ffcmm[m] = pair(t.cmm[m]);
        t.ffcm1[m] = pair(t.cm1[m]);
      }
  }

  template <typename T>
  struct LegT;
  template <>
  struct LegT<double>
  {
    __device__ static double cmm(int m) { return c_leg.cmm[m]; }
    __device__ static double cm1(int m) { return c_leg.cm1[m]; }
    __device__ static double ra(int n, int m) { return c_leg.ra[n][m]; }
    __device__ static double rb(int n, int m) { return c_leg.rb[n][m]; }
  };
  template <>
  struct LegT<float>
  {
    __device__ static float cmm(int m) { return c_leg.fcmm[m]; }
    __device__ static float cm1(int m) { return c_leg.fcm1[m]; }
    __device__ static float ra(int n, int m) { return c_leg.fra[n][m]; }
    __device__ static float rb(int n, int m) { return c_leg.frb[n][m]; }
  };
} // namespace pibem
