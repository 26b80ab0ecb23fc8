// los_fast.cuh -- FP32 line-of-sight integrals of the 3-D functions for the
// fast path: adaptive 21-point Gauss-Kronrod, global bisection of the panel
// with the largest |K21 - G10| until the sum of those differences is below
// kLosEpsRelFast of the integral, at most 32 panels.
//
// One thread per (pixel, component) while a pixel has at most kLosThreadPanels
// panels: neighbouring pixels need nearly the same ones (an edge-on disk 3.5
// on average, 4.5 evaluated), so all lanes do integrand arithmetic.  The few
// pixels that need more are finished by their warp, a lane per node: a thread
// alone would take 100 us for 32 panels, and with it the kernel (that disk's
// values: 92 us with threads alone, 98 with kLosThreadPanels = 8, where the
// 1 % beyond it lie together along the disk's minor axis, 42 with 12, 43 with
// 16).  A warp per pixel throughout left 11 lanes idle and spent three
// quarters of its instructions on shuffle sums: 264 us for the values and 381
// us for the gradient of a 512 x 512 disk + bar; a thread per pixel throughout
// 92 and 180 us, most of it waiting for the last pixels.
//
// Integrands and their analytic parameter derivatives:
//   ExponentialDisk3D  J_0 exp(-R/h) sech^(2/n)(n |z| / (2 z_0))    (function_objects/func_expdisk3d.cpp:226-266)
//   FerrersBar3D       J_0 (1 - m^2)^n inside the ellipsoid m^2 < 1  (function_objects/func_ferrersbar3d.cpp:230-258)
// along s with y_d = yp cos(i) + s sin(i), z_d = yp sin(i) - s cos(i).
// Initial panels: ExponentialDisk3D over [-20h, 20h] split where y_d = 0
// (the radial cusp) and where z_d = 0 (the vertical peak); FerrersBar3D over
// the exact chord of the ellipsoid (m^2 is quadratic in s), where the
// integrand is smooth, so integer n needs a single panel.  The reference's
// QAGS with epsrel 1e-6 integrates over the fixed ranges instead; both are
// integrals of the same function.  The derivative of the integration range
// (20h) is not included: the integrand is below e^-20 of its peak there.
#pragma once
#include "common.cuh"

namespace imfit {

constexpr float kLosEpsRelFast = 4e-6f;
constexpr int kLosMaxPanels = 32;
constexpr int kLosThreadPanels = 12;
constexpr int kLosGrad = 10;  // X0, Y0 and up to 8 function parameters
constexpr float kLog2eF = 1.4426950408889634f;
constexpr float kLn2F = 0.6931471805599453f;
constexpr float kDeg2RadF = 0.017453292519943295f;

// ------------------------------------------------------------ integrands
__device__ __forceinline__ float expdisk_f(const CompF32 &c, float xp, float yp, float s) {
  const float yd = fmaf(s, c.s4, yp * c.s3);
  const float zd = fmaf(-s, c.s3, yp * c.s4);
  const float R = fast_sqrt(fmaf(xp, xp, yd * yd));
  const float u = fabsf(zd) * c.s6;
  const float e2u = fast_ex2(-2.f * kLog2eF * u);
  // log2 sech^alpha(u) = alpha (1 - u log2 e - log2(1 + e^-2u))
  const float l2V = c.s5 * (1.f - u * kLog2eF - fast_lg2(1.f + e2u));
  return c.s0 * fast_ex2(fmaf(-R * c.s1, kLog2eF, l2V));
}

__device__ __forceinline__ float ferrers_f(const CompF32 &c, float xp, float yp, float s) {
  const float yd = fmaf(s, c.s4, yp * c.s3);
  const float zd = fmaf(-s, c.s3, yp * c.s4);
  const float xb = fmaf(xp, c.s5, yd * c.s6);
  const float yb = fmaf(-xp, c.s6, yd * c.s5);
  const float m2 = fmaf(yb * yb, c.subScale, fmaf(xb * xb, c.subInner, zd * zd * c.subSmallK));
  if (!(m2 < 1.f)) return 0.f;
  return c.s0 * fast_ex2(c.s7 * fast_lg2(1.f - m2));
}

// value and d/d(X0, Y0, PA, inc, barPA, J_0, R_bar, q, q_z, n)
__device__ __forceinline__ float ferrers_fg(const CompF32 &c, float xp, float yp, float s, float *g) {
  const float ci = c.s3, si = c.s4, cb = c.s5, sb = c.s6;
  const float ia2 = c.subScale, ib2 = c.subInner, ic2 = c.subSmallK, n = c.s7;
  const float yd = fmaf(s, si, yp * ci);
  const float zd = fmaf(-s, ci, yp * si);
  const float xb = fmaf(xp, cb, yd * sb);
  const float yb = fmaf(-xp, sb, yd * cb);
  const float m2 = fmaf(yb * yb, ia2, fmaf(xb * xb, ib2, zd * zd * ic2));
  if (!(m2 < 1.f)) {
#pragma unroll
    for (int q = 0; q < kLosGrad; q++) g[q] = 0.f;
    return 0.f;
  }
  const float lW = fast_lg2(1.f - m2);
  const float P = fast_ex2(n * lW);
  const float f = c.s0 * P;
  const float fm = -n * c.s0 * fast_ex2((n - 1.f) * lW);  // df/dm^2
  const float dxb = 2.f * xb * ib2 * fm, dyb = 2.f * yb * ia2 * fm;
  const float fxp = fmaf(dxb, cb, -dyb * sb);
  const float fyd = fmaf(dxb, sb, dyb * cb);
  const float fzd = 2.f * zd * ic2 * fm;
  const float gp = fmaf(fyd, ci, fzd * si);
  g[0] = fmaf(-c.cosPA, fxp, c.sinPA * gp);
  g[1] = fmaf(-c.sinPA, fxp, -c.cosPA * gp);
  g[2] = kDeg2RadF * fmaf(fxp, yp, -gp * xp);
  g[3] = kDeg2RadF * fmaf(fyd, fmaf(s, ci, -yp * si), fzd * fmaf(yp, ci, s * si));
  g[4] = kDeg2RadF * 2.f * fm * xb * yb * (ib2 - ia2);
  g[5] = P;
  g[6] = fm * (-2.f * m2 * __fdividef(1.f, c.s1));
  g[7] = fm * (-2.f * xb * xb * ib2 * __fdividef(1.f, c.s2));
  g[8] = fm * (-2.f * zd * zd * ic2 * __fdividef(1.f, c.pad));
  g[9] = f * lW * kLn2F;
  return f;
}

// number of function parameters of a 3-D component
__device__ __forceinline__ int los_nparams(const CompF32 &c) { return c.type == F_EXPDISK3D ? 6 : 8; }

// ------------------------------------------------------------- the rule
// GK21_XGK, GK21_WGK and GK21_WG (gk21_nodes.cuh) rounded to FP32: abscissae
// pairs +-kGkX[k], Kronrod weights, Gauss weights (0 at the Kronrod-only nodes);
// entry 10 is the centre.
__device__ __constant__ float kGkX[11] = {
    9.9565716302580808e-1f, 9.7390652851717172e-1f, 9.3015749135570823e-1f, 8.6506336668898451e-1f,
    7.8081772658641690e-1f, 6.7940956829902441e-1f, 5.6275713466860468e-1f, 4.3339539412924719e-1f,
    2.9439286270146020e-1f, 1.4887433898163121e-1f, 0.0f};
__device__ __constant__ float kGkW[11] = {
    1.1694638867371874e-2f, 3.2558162307964727e-2f, 5.4755896574351996e-2f, 7.5039674810919953e-2f,
    9.3125454583697606e-2f, 1.0938715880229764e-1f, 1.2349197626206585e-1f, 1.3470921731147333e-1f,
    1.4277593857706008e-1f, 1.4773910490133849e-1f, 1.4944555400291691e-1f};
__device__ __constant__ float kGkG[11] = {
    0.f, 6.6671344308688138e-2f, 0.f, 1.4945134915058059e-1f, 0.f, 2.1908636251598204e-1f, 0.f,
    2.6926671930999636e-1f, 0.f, 2.9552422471475287e-1f, 0.f};

template <bool DISK>
__device__ __forceinline__ float los_f(const CompF32 &c, float xp, float yp, float s) {
  return DISK ? expdisk_f(c, xp, yp, s) : ferrers_f(c, xp, yp, s);
}

template <bool DISK>
__device__ __forceinline__ void los_panel(const CompF32 &c, float xp, float yp, float lo, float hi, float &res,
                                          float &err) {
  const float mid = 0.5f * (lo + hi), half = 0.5f * (hi - lo);
  float K = kGkW[10] * los_f<DISK>(c, xp, yp, mid), G = 0.f;
#pragma unroll
  for (int k = 0; k < 10; k++) {
    const float dx = half * kGkX[k];
    const float f = los_f<DISK>(c, xp, yp, mid - dx) + los_f<DISK>(c, xp, yp, mid + dx);
    K = fmaf(kGkW[k], f, K);
    if (k & 1) G = fmaf(kGkG[k], f, G);
  }
  res = K * half;
  err = fabsf((K - G) * half);
}

// The same panel by a whole warp, a lane per node (all lanes hold the result).
__device__ __forceinline__ float los_wsum(float v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <bool DISK>
__device__ __forceinline__ void los_panel_warp(const CompF32 &c, float xp, float yp, float lo, float hi, float &res,
                                               float &err) {
  const int lane = threadIdx.x & 31, k = lane < 10 ? lane : (lane < 20 ? lane - 10 : 10);
  const float mid = 0.5f * (lo + hi), half = 0.5f * (hi - lo);
  const float dx = half * kGkX[k];
  const float f = lane < 21 ? los_f<DISK>(c, xp, yp, lane < 10 ? mid - dx : mid + dx) : 0.f;
  const float K = los_wsum(kGkW[k] * f), G = los_wsum(kGkG[k] * f);
  res = K * half;
  err = fabsf((K - G) * half);
}

// A thread's partition of one pixel's line of sight.
struct LosPanels {
  float lo[kLosThreadPanels], hi[kLosThreadPanels], res[kLosThreadPanels], err[kLosThreadPanels];
};

// Returns the number of panels (0 when the integrand is zero everywhere) and
// the integral in total; more: the tolerance tol needs more than
// kLosThreadPanels (los_finish_warp goes on from P).
//
// tol is kLosEpsRelFast or, for lines that graze the bar, the rounding of the
// integrand itself: 1 - m^2 carries about four units of FP32 rounding of 1, so
// with W its largest value on the line, (1 - m^2)^n is known to 5e-7 n / W of
// itself, and bisecting below that splits a panel into 32 for nothing -- at
// the bar's outline, where the values are smallest (72 us instead of 43 for
// the values of the 512 x 512 disk + bar, the same image to 1e-9).
template <bool DISK>
__device__ __forceinline__ int los_partition(const CompF32 &c, float xp, float yp, LosPanels &P, float &total,
                                             bool &more, float &tol) {
  more = false;
  tol = kLosEpsRelFast;
  float a, b, bp[2] = {0.f, 0.f};
  int nbp = 0;
  if (DISK) {
    b = c.subInner;
    a = -b;
    const float ci = c.s3, si = c.s4;
    if (si > 1e-6f) {
      const float t = -yp * ci / si;  // y_d = 0
      if (t > a && t < b) bp[nbp++] = t;
    }
    if (ci > 1e-6f) {
      const float t = yp * si / ci;  // z_d = 0
      if (t > a && t < b) {
        if (nbp) bp[1] = t;
        else bp[0] = t;
        nbp++;
      }
    }
    if (nbp == 2) {
      if (bp[0] > bp[1]) {
        const float t = bp[0];
        bp[0] = bp[1];
        bp[1] = t;
      }
      if (!(bp[1] > bp[0])) nbp = 1;
    }
  } else {
    // chord of the ellipsoid: m^2(s) = A s^2 + 2 B s + C
    const float ci = c.s3, si = c.s4, cb = c.s5, sb = c.s6;
    const float ia2 = c.subScale, ib2 = c.subInner, ic2 = c.subSmallK;
    const float yd0 = yp * ci, zd0 = yp * si;
    const float xb0 = fmaf(xp, cb, yd0 * sb), xb1 = si * sb;
    const float yb0 = fmaf(-xp, sb, yd0 * cb), yb1 = si * cb;
    const float z1 = -ci;
    const float A = fmaf(yb1 * yb1, ia2, fmaf(xb1 * xb1, ib2, z1 * z1 * ic2));
    const float B = fmaf(yb0 * yb1, ia2, fmaf(xb0 * xb1, ib2, zd0 * z1 * ic2));
    const float C = fmaf(yb0 * yb0, ia2, fmaf(xb0 * xb0, ib2, zd0 * zd0 * ic2));
    const float D = fmaf(B, B, -A * (C - 1.f));
    if (!(A > 0.f) || !(D > 0.f)) {
      total = 0.f;
      return 0;
    }
    tol = fmaxf(tol, 5e-7f * c.s7 * A / D);  // W = D / A
    const float sq = sqrtf(D);
    const float qv = -(B + copysignf(sq, B));
    float s1 = qv / A, s2 = (qv != 0.f) ? (C - 1.f) / qv : -s1;
    if (s1 > s2) {
      const float t = s1;
      s1 = s2;
      s2 = t;
    }
    const float L = c.q;
    a = fmaxf(s1, -L);
    b = fminf(s2, L);
    if (!(b > a)) {
      total = 0.f;
      return 0;
    }
  }
  // one panel per round -- the pieces between the breakpoints, then the halves
  // of the worst panel -- so that the integrand's code is there once and the
  // lanes stay together although their pixels are at different steps
  int np = 0, id = 0;
  float lo = a, hi = nbp ? bp[0] : b, next = 0.f;  // next: the end of the other half, where one waits
  bool half = false;
  for (;;) {
    float r, e;
    los_panel<DISK>(c, xp, yp, lo, hi, r, e);
    P.lo[id] = lo;
    P.hi[id] = hi;
    P.res[id] = r;
    P.err[id] = e;
    if (half) {  // the second half of the bisected panel
      half = false;
      lo = hi;
      hi = next;
      id = np++;
      continue;
    }
    if (np <= nbp) {  // another piece?
      np++;
      if (np <= nbp) {
        lo = hi;
        hi = np < nbp ? bp[1] : b;
        id = np;
        continue;
      }
    }
    float tot = 0.f, etot = 0.f, worst = -1.f;
    for (int i = 0; i < np; i++) {
      const float v = P.err[i];
      tot += P.res[i];
      etot += v;
      if (v > worst) {
        worst = v;
        id = i;
      }
    }
    total = tot;
    if (!(etot > tol * fabsf(tot))) break;
    if (np >= kLosThreadPanels) {
      more = true;
      break;
    }
    lo = P.lo[id];
    next = P.hi[id];
    hi = 0.5f * (lo + next);
    if (!(hi > lo && hi < next)) break;
    half = true;
  }
  return np;
}

// The warp finishes lane src's pixel: lane i < np ends up with panel i in lo,
// hi; returns np, the integral in total (every lane).
template <bool DISK>
__device__ __forceinline__ int los_finish_warp(const CompF32 &c, float xp, float yp, const LosPanels &P, float tol,
                                               int src, float &lo, float &hi, float &total) {
  const int lane = threadIdx.x & 31;
  float res = 0.f, err = 0.f;
  tol = __shfl_sync(0xffffffffu, tol, src);
  int np = kLosThreadPanels;
  lo = hi = 0.f;
#pragma unroll
  for (int i = 0; i < kLosThreadPanels; i++) {
    const float l = __shfl_sync(0xffffffffu, P.lo[i], src), h = __shfl_sync(0xffffffffu, P.hi[i], src);
    const float r = __shfl_sync(0xffffffffu, P.res[i], src), e = __shfl_sync(0xffffffffu, P.err[i], src);
    if (lane == i) {
      lo = l;
      hi = h;
      res = r;
      err = e;
    }
  }
  for (;;) {
    const float tot = los_wsum(res), etot = los_wsum(err);
    total = tot;
    if (!(etot > tol * fabsf(tot)) || np >= kLosMaxPanels) break;
    float e = lane < np ? err : -1.f;
    int id = lane;
    for (int o = 16; o > 0; o >>= 1) {
      const float e2 = __shfl_xor_sync(0xffffffffu, e, o);
      const int i2 = __shfl_xor_sync(0xffffffffu, id, o);
      if (e2 > e || (e2 == e && i2 < id)) {
        e = e2;
        id = i2;
      }
    }
    const float plo = __shfl_sync(0xffffffffu, lo, id), phi = __shfl_sync(0xffffffffu, hi, id);
    const float m = 0.5f * (plo + phi);
    if (!(m > plo && m < phi)) break;
    float r1, e1, r2, e2;
    los_panel_warp<DISK>(c, xp, yp, plo, m, r1, e1);
    los_panel_warp<DISK>(c, xp, yp, m, phi, r2, e2);
    if (lane == id) {
      hi = m;
      res = r1;
      err = e1;
    }
    if (lane == np) {
      lo = m;
      hi = phi;
      res = r2;
      err = e2;
    }
    np++;
  }
  return np;
}

// Adds r times the derivative integrals over one panel of the disk to acc: d/d(X0,
// Y0, PA, inc, J_0, h, n, z_0).  With E the density over J_0, and everything that
// is constant along the line of sight (the rotation, the scale factors) kept
// out of the nodes, eight sums hold all of them: in terms of
//   q = E / R,  t = E sgn(z_d) tanh u  (f_R = -J_0 E / h, f_z = -J_0 t / z_0)
// sum q, q y_d, t, q y_d z_d / h - t y_d / z_0, E, E R, E (u tanh u - ln cosh u),
// E u tanh u.  42 instructions a node instead of 75.
__device__ __forceinline__ void expdisk_grad_panel(const CompF32 &c, float xp, float yp, float lo, float hi, float r,
                                                   float *acc) {
  const float ci = c.s3, si = c.s4, alpha = c.s5, ih = c.s1, iz0 = c.s6 * c.s5;  // 1/z_0 = alpha / (alpha z_0)
  const float mid = 0.5f * (lo + hi), half = 0.5f * (hi - lo);
  const float yd0 = yp * ci, zd0 = yp * si, x2 = xp * xp;
  float sq = 0.f, sqy = 0.f, st = 0.f, si_ = 0.f, sE = 0.f, sER = 0.f, sn = 0.f, sz = 0.f;
#pragma unroll 2
  for (int k = 0; k < 21; k++) {  // the pairs, then the centre
    const int j = k >> 1;
    const float dx = half * kGkX[j];
    const float s = (k & 1) ? mid + dx : mid - dx;
    const float yd = fmaf(s, si, yd0), zd = fmaf(-s, ci, zd0);
    const float R = fast_sqrt(fmaf(yd, yd, x2));
    const float Rinv = R > 0.f ? __fdividef(1.f, R) : 0.f;
    const float u = fabsf(zd) * c.s6;
    const float e2u = fast_ex2(-2.f * kLog2eF * u);
    const float th = __fdividef(1.f - e2u, 1.f + e2u);
    const float l2c = 1.f - u * kLog2eF - fast_lg2(1.f + e2u);  // -log2 cosh u
    const float E = kGkW[j] * fast_ex2(fmaf(-R * ih, kLog2eF, alpha * l2c));
    const float q = E * Rinv, qy = q * yd;
    const float t = zd != 0.f ? copysignf(E * th, zd) : 0.f;
    const float uth = u * th;
    sq += q;
    sqy += qy;
    st += t;
    si_ = fmaf(qy, zd * ih, fmaf(-t * iz0, yd, si_));
    sE += E;
    sER = fmaf(E, R, sER);
    sn = fmaf(E, fmaf(kLn2F, l2c, uth), sn);
    sz = fmaf(E, uth, sz);
  }
  r *= half;
  const float f = r * c.s0;
  const float fx = -f * ih * xp * sq;                      // sum of f_x'
  const float gp = -f * fmaf(ih * ci, sqy, iz0 * si * st);  // sum of f_yd cos i + f_zd sin i
  acc[0] = fmaf(-c.cosPA, fx, fmaf(c.sinPA, gp, acc[0]));
  acc[1] = fmaf(-c.sinPA, fx, fmaf(-c.cosPA, gp, acc[1]));
  acc[2] = fmaf(kDeg2RadF, fmaf(fx, yp, -gp * xp), acc[2]);
  acc[3] = fmaf(kDeg2RadF * f, si_, acc[3]);
  acc[4] = fmaf(r, sE, acc[4]);
  acc[5] = fmaf(f * ih * ih, sER, acc[5]);
  acc[6] = fmaf(f * (-0.5f * alpha * alpha), sn, acc[6]);
  acc[7] = fmaf(f * alpha * iz0, sz, acc[7]);
}

// Adds r times the derivative integrals over one panel to acc[0..kLosGrad).
template <bool DISK>
__device__ __forceinline__ void los_grad_panel(const CompF32 &c, float xp, float yp, float lo, float hi, float r,
                                               float *acc) {
  if (DISK) {
    expdisk_grad_panel(c, xp, yp, lo, hi, r, acc);
    return;
  }
  const float mid = 0.5f * (lo + hi), half = 0.5f * (hi - lo);
  r *= half;
#pragma unroll 2
  for (int k = 0; k < 21; k++) {
    const int j = k >> 1;
    const float dx = half * kGkX[j];
    float t[kLosGrad];
    ferrers_fg(c, xp, yp, (k & 1) ? mid + dx : mid - dx, t);
    const float w = r * kGkW[j];
#pragma unroll
    for (int q = 0; q < kLosGrad; q++) acc[q] = fmaf(w, t[q], acc[q]);
  }
}

}  // namespace imfit
