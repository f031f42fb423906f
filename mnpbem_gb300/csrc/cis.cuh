// exp(i k d) in FP64 for kernels that evaluate it per pair: table-driven, in
// shared memory (see cis_exp).  The table lives in assemble.cu.
#pragma once
#include "common.cuh"

namespace mnpbem {

// ------------------------------------------------------- exp(i k d), FP64
// Table-driven evaluation (Cody-Waite argument reduction + short Taylor
// polynomials), a few FP64 FMAs per call instead of a library sincos and exp:
//   phase  th = Re(k) d = j (2 pi / 256) + t,  |t| <= pi / 256:
//          cis(th) = cis(2 pi j / 256) * (cos t + i sin t), Taylor to t^8;
//   decay  x = Im(k) d = y (ln 2 / 64) + u,   |u| <= ln 2 / 128:
//          exp(-x) = 2^(-floor(y/64)) * 2^(-(y mod 64)/64) * exp(-u), Taylor to u^7.
// The reduction constants are split in a 32-bit head (exact products with
// |j| < 2^20) and a tail; the tables come from the device's sincospi / exp2
// once per device.  Accuracy: a few ulp of the FP64 result.
constexpr int CIS_N = 256;
constexpr double CIS_INV = 40.74366543152521;        // 256 / (2 pi)
constexpr double CIS_C1 = 0.024543692605220713;      // 2 pi / 256, head
constexpr double CIS_C2 = 9.495469541415925e-13;     // 2 pi / 256, tail
constexpr double EXP_INV = 92.33248261689366;        // 64 / ln 2
constexpr double EXP_L1 = 0.01083042469326756;       // ln 2 / 64, head
constexpr double EXP_L2 = 2.9815858269852933e-12;    // ln 2 / 64, tail

struct CisTable {
  double2 cs[CIS_N];   // (cos, sin)(2 pi j / 256)
  double e2[64];       // 2^(-m / 64)
};
// device address of the table (filled on the device's first call)
mnpbem_status cis_table(const CisTable** table, cudaStream_t st);

// copy into shared memory; every thread of the block calls it (it ends in a barrier)
__device__ __forceinline__ void cis_load(CisTable& t, const CisTable* src) {
  for (int q = threadIdx.x; q < CIS_N; q += blockDim.x) t.cs[q] = src->cs[q];
  for (int q = threadIdx.x; q < 64; q += blockDim.x) t.e2[q] = src->e2[q];
  __syncthreads();
}

// exp(i k d) for complex k (Im k >= 0 for passive media; any sign works: 0 beyond a decay
// of exp(-700), infinite where the growth leaves the range).  SHIFT:
// j by adding 1.5 2^52, whose low word is j (two FP64 operations instead of a
// product, a rounding and a conversion; the last bits may differ, as a phase next to
// the middle of two table entries may go to the other)
template <bool SHIFT = false>
__device__ __forceinline__ double2 cis_exp(const CisTable& T, double2 k, double d) {
  const double th = k.x * d;
  double jf;
  int j;
  if constexpr (SHIFT) {
    const double jm = fma(th, CIS_INV, 6755399441055744.0);
    j = __double2loint(jm);
    jf = jm - 6755399441055744.0;
  } else {
    jf = rint(th * CIS_INV);
    j = (int)((long long)jf & (CIS_N - 1));
  }
  const double t = fma(-jf, CIS_C2, fma(-jf, CIS_C1, th));
  const double t2 = t * t;
  const double sn = t * fma(t2, fma(t2, fma(t2, -1.0 / 5040.0, 1.0 / 120.0), -1.0 / 6.0), 1.0);
  const double cn = fma(t2, fma(t2, fma(t2, fma(t2, 1.0 / 40320.0, -1.0 / 720.0), 1.0 / 24.0), -0.5), 1.0);
  const double2 tb = T.cs[j & (CIS_N - 1)];
  double cr = tb.x * cn - tb.y * sn;
  double sr = fma(tb.y, cn, tb.x * sn);
  if (k.y != 0.0) {
    const double x = k.y * d;
    double e;
    if (x > 700.0) {
      e = 0.0;
    } else {
      const double yf = rint(x * EXP_INV);
      const double u = fma(-yf, EXP_L2, fma(-yf, EXP_L1, x));
      const double v = -u;
      const double ev = fma(v, fma(v, fma(v, fma(v, fma(v, fma(v, fma(v, 1.0 / 5040.0, 1.0 / 720.0), 1.0 / 120.0),
                                                          1.0 / 24.0), 1.0 / 6.0), 0.5), 1.0), 1.0);
      const long long yi = (long long)yf;
      const long long nn = yi >> 6;                 // floor(y / 64)
      const int m = (int)(yi - (nn << 6));
      e = ev * T.e2[m];
      if (nn > -1000) {
        e *= __longlong_as_double((unsigned long long)(1023 - nn) << 52);   // 2^(-nn)
      } else {         // growth to the end of the range and beyond (infinity)
        const long long up = nn < -2023 ? 1023 : -nn - 1000;
        e = e * __longlong_as_double((long long)(1023 + 1000) << 52) * __longlong_as_double((1023 + up) << 52);
      }
    }
    cr *= e;
    sr *= e;
  }
  return make_double2(cr, sr);
}

}  // namespace mnpbem
