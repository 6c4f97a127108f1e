// hc3d_lucy.cuh -- the Lucy temperature of one cell and species, shared by
// every kernel that solves it: tfinal (the module is not shipped; restated as
// the fixed point of dusttemp.f90:30-50 with the absorbed-path estimator in
// place of the absorption count), with KapP (dust.f90:114-141).
#pragma once

#include <cuda_runtime.h>

namespace hc3d {

// What bounds the solve is the FP64 pipe (1/64 of the FP32 rate on this GPU):
// some eight steps per cell, each a logarithm for the opacity's row and a fourth
// root. log(), pow() and the divisions made 190 FP64 instructions of a step.
// The fourth root of a cell's constant factor is formed once and that of the
// opacity by a cubic correction of an FP32 root, the rows' reciprocal spacings
// are kept in shared memory, and the logarithm is table-driven: about 35, and
// 18.3 ms against 71.0 for the 20.7 million (cell, species) pairs of the
// full-3D grid (hc3d_lucy_update_noalloc), 0.83 GB of inputs and outputs.
//
// The logarithm: P.T.P. Tang, "Table-driven implementation of the logarithm
// function in IEEE floating-point arithmetic", ACM TOMS 16 (1990) 378. x = 2^e
// m, m in [1, 2); with F the mid-point of m's interval of 1/128 and r = m/F - 1
// (|r| < 1/256), log x = e ln 2 + log F + log(1 + r), the last by its series up
// to r^7 (the next term is below 2^-67).
constexpr int kLucyLog = 128;   // intervals of the logarithm's table
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
  const int e = (int)(hi >> 20) - 1023, i = (int)(hi >> 13) & (kLucyLog - 1);
  const double m = __hiloint2double((int)((hi & 0xfffffu) | 0x3ff00000u), __double2loint(x));
  const double r = fma(m, q.rcp[i], -1.0);
  double s = fma(r, 1.0 / 7.0, -1.0 / 6.0);
  s = fma(s, r, 1.0 / 5.0);
  s = fma(s, r, -1.0 / 4.0);
  s = fma(s, r, 1.0 / 3.0);
  s = fma(s, r, -1.0 / 2.0);
  s = fma(s * r, r, r);
  return fma((double)e, 0.693147180559945309417232121458, q.logf[i] + s);
}

// KapP: Planck-mean kappa/kappa_V at T (K/11605), linear in log T.
__device__ __forceinline__ double lucy_kapp(const LucyTables& q, const double* lTint, int nT, const double* kp,
                                            double l1, double rl, double T) {
  const double lT = lucy_log(q, T);
  const int k = (int)((lT - l1) * rl) + 1;
  if (k < 1) return kp[0];
  if (k > nT - 1) return kp[nT - 1];
  const double d = lT - lTint[k - 1];
  const double f = k <= kLucyRows ? d * q.rdl[k - 1] : d / (lTint[k] - lTint[k - 1]);
  return (1.0 - f) * kp[k - 1] + f * kp[k];
}

// x^(-1/4): an FP32 root, then one step of third order. With x y^4 = 1 - h, h
// about 1e-6 of FP32 rounding, x^(-1/4) = y (1 + h/4 + 5 h^2/32 + O(h^3)).
__device__ __forceinline__ double lucy_root4_inv(double x) {
  if (!(x > 1e-30 && x < 1e30)) return 1.0 / sqrt(sqrt(x));  // outside FP32
  const double y = (double)rsqrtf(sqrtf((float)x));
  const double y2 = y * y;
  const double h = fma(-x, y2 * y2, 1.0);
  return fma(y * h, fma(h, 5.0 / 32.0, 0.25), y);
}

// Energy balance 4 sigma T^4 kappa_V kappa_P(T) (rho V) = na L / N, iterated
// from T0 to 1e-5 relative (at most 1000 steps), clamped to [0.1, 1600] K.
__device__ __forceinline__ double lucy_dusttemp(const LucyTables& q, const double* lTint, int nT, const double* kp,
                                                double kappav, double ltot, double nphot, double na, double T0,
                                                double massarr) {
  const double eps = 1.e-5, sigt = 5.670400e-5, lo = 0.1 / 11605.0, hi = 1600.0 / 11605.0;
  const double l1 = lTint[0], rl = (double)(nT - 1) / (lTint[nT - 1] - l1);
  const double c = (na * ltot) / (4.0 * sigt * nphot * kappav);
  const double g = sqrt(sqrt(c)) / (11605.0 * massarr);
  double Td = T0 != 0.0 ? T0 : lo;
  if (Td < 0.0) return __longlong_as_double(0x7ff8000000000000ll);  // its logarithm
  double Told = 0.5 * Td;
  int it = 0;
  while (fabs(Td - Told) > eps * Td && it < 1000) {
    ++it;
    Told = Td;
    const double r = lucy_root4_inv(lucy_kapp(q, lTint, nT, kp, l1, rl, Td));
    Td = massarr > 0.0 ? r * g : lo;  // no mass: the floor
    if (Td > hi) Td = hi;
    if (Td < lo) Td = lo;
  }
  return Td;
}

}  // namespace hc3d
