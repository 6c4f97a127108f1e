// hc3d_lucy.cuh -- the Lucy temperature of one cell and species, shared by
// every kernel that solves it: tfinal (the module is not shipped; restated as
// the fixed point of dusttemp.f90:30-50 with the absorbed-path estimator in
// place of the absorption count), with KapP (dust.f90:114-141).
#pragma once

#include <cuda_runtime.h>

namespace hc3d {

// What bounds the solve is the FP64 pipe (1/64 of the FP32 rate on this GPU):
// some seven steps per cell, each a logarithm for the opacity's row and a fourth
// root. log(), pow() and the divisions made 190 FP64 instructions of a step,
// 71.0 ms for the 20.7 million (cell, species) pairs of the full-3D grid
// (hc3d_lucy_update_noalloc; 0.83 GB of inputs and outputs). The cell's constants
// are one factor w, so that a step is T = (kappa_P(T) w)^(-1/4): a table-driven
// logarithm, a row, and a cubic correction of an FP32 root; what only orders
// positive numbers is compared as integers, off that pipe. 26 instructions a
// step, and some 30 a cell besides, 13.7 ms (18.3 with the factor's two roots and
// divisions, 128 intervals and the tables formed in each of 20000 blocks).
//
// The logarithm: P.T.P. Tang, "Table-driven implementation of the logarithm
// function in IEEE floating-point arithmetic", ACM TOMS 16 (1990) 378. x = 2^e
// m, m in [1, 2); with F the mid-point of m's interval of 1/1024 and r = m/F - 1
// (|r| < 1/2048), log x = e ln 2 + log F + log(1 + r), the last by its series up
// to r^4 (the next term is below 2^-57, and |log x| above 1.9 over the range of
// temperatures).
//
// Against the same iteration in extended precision the relative error is 1.10e-16
// root mean square over temperatures of 10 to 1500 K; log() and pow() made
// 1.25e-16.  Against an FP64 evaluation in their order, whose roundings it does not
// share, it is 1.2e-16 where theirs was 6.5e-17.
constexpr int kLucyLog = 1024;  // intervals of the logarithm's table
constexpr int kLucyRows = 1024; // opacity rows whose reciprocal spacing is kept in shared memory

struct LucyTables {
  double rcp[kLucyLog], logf[kLucyLog];  // 1/F and -log(1/F)
  double rdl[kLucyRows];                 // 1 / (lTint(k+1) - lTint(k))
};

// every thread of the block, before the first solve
__device__ __forceinline__ void lucy_tables(LucyTables& q, const double* lTint, int nT) {
  for (int i = threadIdx.x; i < kLucyLog; i += blockDim.x) {
    const double c = 1.0 / (1.0 + ((double)i + 0.5) / kLucyLog);
    q.rcp[i] = c;
    q.logf[i] = -log(c);
  }
  for (int i = threadIdx.x; i < min(nT - 1, kLucyRows); i += blockDim.x) q.rdl[i] = 1.0 / (lTint[i + 1] - lTint[i]);
  __syncthreads();
}

// log of a positive normal x
__device__ __forceinline__ double lucy_log(const LucyTables& q, double x) {
  const unsigned hi = (unsigned)__double2hiint(x);
  const int e = (int)(hi >> 20) - 1023, i = (int)(hi >> 10) & (kLucyLog - 1);
  const double m = __hiloint2double((int)((hi & 0xfffffu) | 0x3ff00000u), __double2loint(x));
  const double r = fma(m, q.rcp[i], -1.0);
  double s = fma(r, -1.0 / 4.0, 1.0 / 3.0);
  s = fma(s, r, -1.0 / 2.0);
  s = fma(s * r, r, r);
  return fma((double)e, 0.693147180559945309417232121458, q.logf[i] + s);
}

// KapP: Planck-mean kappa/kappa_V at T (K/11605), linear in log T; row0 = -lTint(1) rl
__device__ __forceinline__ double lucy_kapp(const LucyTables& q, const double* lTint, int nT, const double* kp,
                                            double row0, double rl, double T) {
  const double lT = lucy_log(q, T);
  const int k = (int)fma(lT, rl, row0) + 1;
  if (k < 1) return kp[0];
  if (k > nT - 1) return kp[nT - 1];
  const double d = lT - lTint[k - 1], k0 = kp[k - 1];
  const double f = k <= kLucyRows ? d * q.rdl[k - 1] : d / (lTint[k] - lTint[k - 1]);
  return fma(f, kp[k] - k0, k0);
}

// ltot / (4 sigma N kappa_V): the factor of the absorbed path in the balance
inline double lucy_factor(double ltot, double nphot, double kappav) {
  return ltot / (4.0 * 5.670400e-5 * nphot * kappav);
}

// Energy balance 4 sigma T^4 kappa_V kappa_P(T) (rho V) = na L / N, iterated
// from T0 to 1e-5 relative (at most 1000 steps), clamped to [0.1, 1600] K;
// factor: lucy_factor of the species.
//
// x^(-1/4): an FP32 root, then one step of third order. With x y^4 = 1 - h, h
// about 1e-6 of FP32 rounding, x^(-1/4) = y (1 + h/4 + 5 h^2/32 + O(h^3)).
__device__ __forceinline__ double lucy_dusttemp(const LucyTables& q, const double* lTint, int nT, const double* kp,
                                                double factor, double na, double T0, double massarr) {
  const double eps = 1.e-5, lo = 0.1 / 11605.0, hi = 1600.0 / 11605.0;
  double Td = T0 != 0.0 ? T0 : lo;
  if (!(fabs(Td) < 1.0 / 0.0)) return Td;
  if (Td < 0.0) Td = 2.2250738585072014e-308;  // below the table, as any start under its first row
  const double rl = (double)(nT - 1) / (lTint[nT - 1] - lTint[0]), row0 = -lTint[0] * rl;
  const double m = 11605.0 * massarr, m2 = m * m;
  const double w = na != 0.0 ? (m2 * m2) / (na * factor) : 1.0 / 0.0;  // without a tally the floor, however small m
  for (int it = 0; it < 1000; ++it) {
    const double Told = Td;
    const double x = lucy_kapp(q, lTint, nT, kp, row0, rl, Td) * w;
    if (!(massarr > 0.0)) {
      Td = lo;  // no mass: the floor
    } else if ((unsigned)(__double2hiint(x) - 0x39c00000) < 0x0c600000u) {  // 2^-99 <= x < 2^99: positive, and FP32's
      const double y = (double)rsqrtf(sqrtf((float)x));
      const double y2 = y * y;
      const double h = fma(-x, y2 * y2, 1.0);
      Td = fma(y * h, fma(h, 5.0 / 32.0, 0.25), y);
      if (__double_as_longlong(Td) > __double_as_longlong(hi)) Td = hi;
      if (__double_as_longlong(Td) < __double_as_longlong(lo)) Td = lo;
    } else {
      Td = 1.0 / sqrt(sqrt(x));
      if (!(Td == Td)) return Td;
      if (Td > hi) Td = hi;
      if (Td < lo) Td = lo;
    }
    if (__double_as_longlong(fabs(Td - Told)) <= __double_as_longlong(eps * Td)) break;
  }
  return Td;
}

// the larger of mx and the relative change |T - T0| / T (bits of NaN are larger
// than any number's); the division only where the change may be the larger
__device__ __forceinline__ double lucy_change(double mx, double T, double T0) {
  const double d = fabs(T - T0);
  if (d <= mx * T) return mx;
  const double v = fabs(d / T);
  return __double_as_longlong(v) > __double_as_longlong(mx) ? v : mx;
}

}  // namespace hc3d
