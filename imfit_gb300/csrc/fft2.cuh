// fft2.cuh -- transforms of n = R1 R2 points in two register passes.
//
// A thread holds a whole length-R1 (then R2) sub-transform in registers, so a
// line goes through shared memory once between the passes instead of once per
// radix-4..9 pass: the multi-pass kernels spent their issue slots on shared
// loads, stores, twiddle loads and index arithmetic, with the FP32 pipe 10 %
// busy.  With n = R2 n1 + n2 and k = k1 + R1 k2:
//   pass 1, thread n2: y[k1] = sum over n1 of x[R2 n1 + n2] W_R1^(n1 k1), times
//                      W_n^(n2 k1), kept at k1 R2' + n2 (R2' = R2 or R2 + 1, odd)
//   pass 2, thread k1: X[k1 + R1 k2] = sum over n2 of y W_R2^(n2 k2)
// The inverse runs the same two passes backwards on the same positions, so a
// convolution needs one buffer and two barriers.
//
// Lengths: R1 and R2 from IMFIT_TWO_PASS_RADICES; a length without such a
// factorisation, or beyond 36 x 36, takes the multi-pass kernels (fft.cuh).
#pragma once
#include "fft.cuh"

namespace imfit {

// Two-pass form of one length: t[k1 P + n2] = W_n^(n2 k1) on the device
// (kernels copy it to shared memory; P = two_pass_pitch(R2)).
struct TwoPass {
  int R1 = 0, R2 = 0;  // 0: the length has none
  const cplx<float> *t = nullptr;
};

// pitch of the intermediate's (and the twiddles') rows of R2 values: odd, so
// that the threads of pass 2 (a row apart) hit distinct banks
__host__ __device__ inline int two_pass_pitch(int R2) { return R2 | 1; }
// entries of the twiddle table, even so that it copies in 16-byte pieces
__host__ __device__ inline int two_pass_table(int R1, int R2) { return (R1 * two_pass_pitch(R2) + 1) & ~1; }

// ------------------------------------------------------------ roots of unity
// cos and sin of 2 pi e / N at compile time: reduction to the first octant,
// Taylor series there.
struct RootCs {
  double c, s;
};
__host__ __device__ constexpr RootCs root_of_unity(int e, int N) {
  e = ((e % N) + N) % N;
  int o = 8 * e / N;                 // octant
  int num = 8 * e - o * N;           // angle = (o + num/N) pi/4
  const bool flip = o & 1;           // reflect odd octants
  if (flip) num = N - num;
  const double x = 0.78539816339744830961566 * num / N, x2 = x * x;
  double c = 0.0, s = 0.0;
  for (int k = 12; k >= 0; k--) {
    c = 1.0 - c * x2 / ((2 * k + 1) * (2 * k + 2));
    s = 1.0 - s * x2 / ((2 * k + 2) * (2 * k + 3));
  }
  s *= x;
  if (flip) o++;
  // angle = o pi/4 -/+ x with o even
  const int q = (o / 2) % 4;
  const double sx = flip ? -s : s;
  switch (q) {
    case 0: return {c, sx};
    case 1: return {-sx, c};
    case 2: return {-c, -sx};
    default: return {sx, -c};
  }
}
template <int N>
struct RootTable {
  float c[N], s[N];
  __host__ __device__ constexpr RootTable() : c(), s() {
    for (int e = 0; e < N; e++) {
      const RootCs r = root_of_unity(e, N);
      c[e] = (float)r.c;
      s[e] = (float)r.s;
    }
  }
};

// z exp(S 2 pi i e / N), e a compile-time value after unrolling
template <int N, int S>
__device__ __forceinline__ cplx<float> rotate(cplx<float> z, int e) {
  e %= N;
  if (e == 0) return z;
  if (4 * e % N == 0) {
    const int q = 4 * e / N;
    if (q == 2) return {-z.x, -z.y};
    return mul_si(z, q == 1 ? S : -S);
  }
  constexpr RootTable<N> w;
  const float c = w.c[e], s = S * w.s[e];
  return {z.x * c - z.y * s, z.x * s + z.y * c};
}

// first factor of the composite sub-transforms
template <int N>
__host__ __device__ constexpr int first_factor() {
  return N == 6 || N == 10 || N == 14 ? 2 : N == 18 ? 2 : N == 12 || N == 15 || N == 21 || N == 24 || N == 27 ? 3
         : N == 16 || N == 20 || N == 28 || N == 32 || N == 36 ? 4 : N == 25 || N == 30 || N == 35 ? 5 : N;
}

// length-N DFT in registers, sign S, natural order in and out: N = A B with
// n = B n1 + n2, k = k1 + A k2
template <int N, int S>
__device__ __forceinline__ void dft_reg(cplx<float> *v) {
  constexpr int A = first_factor<N>();
  if constexpr (N == 2) {
    dft2(v);
  } else if constexpr (N == 3) {
    dft3(v, S);
  } else if constexpr (N == 4) {
    dft4(v, S);
  } else if constexpr (N == 5) {
    dft5(v, S);
  } else if constexpr (N == 7) {
    dft7(v, S);
  } else if constexpr (N == 8) {
    dft8(v, S);
  } else if constexpr (N == 9) {
    dft9(v, S);
  } else {
    constexpr int B = N / A;
    cplx<float> y[N];
#pragma unroll
    for (int n2 = 0; n2 < B; n2++) {
      cplx<float> t[A];
#pragma unroll
      for (int n1 = 0; n1 < A; n1++) t[n1] = v[n2 + B * n1];
      dft_reg<A, S>(t);
#pragma unroll
      for (int k1 = 0; k1 < A; k1++) y[k1 * B + n2] = rotate<N, S>(t[k1], n2 * k1);
    }
#pragma unroll
    for (int k1 = 0; k1 < A; k1++) {
      cplx<float> t[B];
#pragma unroll
      for (int n2 = 0; n2 < B; n2++) t[n2] = y[k1 * B + n2];
      dft_reg<B, S>(t);
#pragma unroll
      for (int k2 = 0; k2 < B; k2++) v[k1 + A * k2] = t[k2];
    }
  }
}

#define IMFIT_TWO_PASS_RADICES(X) \
  X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(12) X(14) X(15) X(16) X(18) X(20) X(21) X(24) X(25) X(27) X(28) X(30) X(32) X(35) X(36)

inline bool two_pass_radix(int r) {
  switch (r) {
#define X(R) case R:
    IMFIT_TWO_PASS_RADICES(X)
    return true;
#undef X
    default: return false;
  }
}

// The factorisation of n with the smallest larger factor (fewest registers,
// most balanced passes), the larger factor first.  Returns false where there
// is none.
inline bool two_pass_factors(int n, int &R1, int &R2) {
  R1 = R2 = 0;
  for (int a = 1; a * a <= n; a++)
    if (n % a == 0 && two_pass_radix(a) && two_pass_radix(n / a)) {
      R1 = n / a;  // the last (largest) a wins
      R2 = a;
    }
  return R1 > 0;
}

}  // namespace imfit
