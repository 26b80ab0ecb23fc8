// fp64_math.cuh -- the plain path's FP64 exp2, log2 and square root, written
// for few FP64 instructions.
//
// GB300 issues two FP64 lanes per SM per clock (measured 2.1; FP32: 128), so a
// warp instruction on the FP64 pipe takes sixteen cycles of its SM and the
// plain path's time is its number of FP64 instructions.  Table lookups and
// integer work are free beside them.  The table-driven forms (Tang, ACM TOMS
// 15 (1989) 144 and 16 (1990) 378; tables and Taylor coefficients from
// gen_fp64_tables.py) take 9 to 10 of them, and carry their arguments as
// unevaluated sums h + l so that exp2(s log2 v) loses nothing in between:
//   log2_hl   |error| < 2^-57 absolute, plus half an ulp of l
//   exp2_hl   < 1 ulp
//   sqrt64    correctly rounded up to the last Newton step's rounding (< 1 ulp)
// Explicit fma() calls only: the units that include this are compiled without
// contraction.
#pragma once
#include <cuda_runtime.h>

#include "fp64_tables.cuh"

namespace imfit {

// Copies of the tables in shared memory (lanes index them at random).
struct Fp64Tables {
  double e2[64];
  double rec[128], lhi[128], llo[128];
};

__device__ __forceinline__ void fp64_tables_load(Fp64Tables &t) {
  for (int i = threadIdx.x; i < 64; i += blockDim.x) t.e2[i] = kExp2Tab[i];
  double *l = t.rec;  // rec, lhi, llo are consecutive
  for (int i = threadIdx.x; i < 3 * 128; i += blockDim.x) l[i] = kLog2Tab[i];
}

struct hl64 {
  double h, l;
};

// log2 of a positive, normal, finite v as h + l (|l| < 2^-7): v = 2^k m,
// f = m c_i - 1 (one fma, |f| <= 2^-8), log2 v = (k + hi_i) + (lo_i + P(f)).
__device__ __forceinline__ hl64 log2_hl(const Fp64Tables &t, double v) {
  const int hi = __double2hiint(v);
  const int i = (hi >> 13) & 127;
  const double m = __hiloint2double((hi & 0xfffff) | 0x3ff00000, __double2loint(v));
  // k as a double: 2^52 + 2^31 + k less the constant
  const double k = __hiloint2double(0x43300000, ((hi >> 20) - 1023) ^ 0x80000000) - 4503601774854144.0;
  const double f = fma(m, t.rec[i], -1.0);
  constexpr double C[6] = IMFIT_LOG2_COEF;
  double p = C[5];
#pragma unroll
  for (int q = 4; q >= 0; q--) p = fma(p, f, C[q]);
  return {k + t.lhi[i], fma(p, f, t.llo[i])};
}

// 2^(h + l), |l| <= 2^-7 (SMALL: |l| < 2^-20): h + l = j/64 + r, 2^(j/64) from
// the table and the exponent, 2^r - 1 by its Taylor polynomial.  Below 2^-1075
// the result is 0; near the ends of the range the library's exp2 gives it.
template <bool SMALL>
__device__ __forceinline__ double exp2_hl(const Fp64Tables &t, double h, double l) {
  const int top = __double2hiint(h);
  if ((top & 0x7fffffff) >= 0x408fe000) {  // |h| >= 1020
    if (top < 0 && h < -1080.0) return 0.0;
    return exp2(h + l);
  }
  const double big = 105553116266496.0;  // 1.5 2^46: multiples of 1/64 in the low word
  const double s = (SMALL ? h : h + l) + big;
  const int j = __double2loint(s);
  const double r = (h - (s - big)) + l;
  constexpr double C[5] = IMFIT_EXP2_COEF;
  double p = C[4];
#pragma unroll
  for (int q = 3; q >= 0; q--) p = fma(p, r, C[q]);
  const double T = t.e2[j & 63];
  const double v = fma(T, p * r, T);
  return __hiloint2double(__double2hiint(v) + ((j >> 6) << 20), __double2loint(v));
}

// s (a.h + a.l) as an unevaluated sum
__device__ __forceinline__ hl64 scale_hl(hl64 a, double s) {
  const double p = s * a.h;
  return {p, fma(s, a.l, fma(s, a.h, -p))};
}

// Square root of a positive, normal, finite v (not near the ends of the
// range): the SFU's reciprocal square root of the high word, one coupled
// Newton step (Goldschmidt's form, two multiplications) and a final
// correction with the exact residual v - s^2.
__device__ __forceinline__ double sqrt64(double v) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
  double s = v * y, hf = 0.5 * y;
  const double e = fma(-s, hf, 0.5);
  s = fma(s, e, s);
  hf = fma(hf, e, hf);
  return fma(fma(-s, s, v), hf, s);
}

}  // namespace imfit
