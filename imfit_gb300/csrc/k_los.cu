// k_los.cu -- plain FP64 line-of-sight integrals of the 3-D functions, one
// thread per (model pixel, 3-D component), QAGS per pixel (qags_dev.cuh).
// Compiled with --fmad=false like the rest of the plain path.
//
//   ExponentialDisk3D  function_objects/func_expdisk3d.cpp:178-266
//   FerrersBar3D       function_objects/func_ferrersbar3d.cpp:172-258,
//                      Compute3dObjectCoords function_objects/helper_funcs_3d.cpp:65-82
//
// FP64-issue bound: an integral takes 21 integrand values per panel, so its
// time is the integrand's FP64 instructions.  The integrands are therefore
// written for few of them (about 50 for the disk and 15 for an integer-index
// bar, with fp64_math.cuh's exp2 and log2, instead of 400 and 130 with cosh,
// pow, exp and five divisions); the same functions to a few units of the last
// place, so QAGS takes the same decisions.
#include "fp64_math.cuh"
#include "kernels.h"
#include "qags_dev.cuh"

namespace imfit {

constexpr double kExpDiskIntegMult = 20.0; // func_expdisk3d.cpp:66
constexpr double kLosEpsRel = 1.0e-6;      // integrator.cpp:39-51
constexpr double kLog2e64 = 1.4426950408889634;

// The reference's expressions of the two densities, for values that come near
// the bottom of the FP64 range (below 2^-900): denormal values have few
// bits, QAGS sees their rounding as structure, and only the same bits give the
// same decisions -- and the same integrals within the device's list of
// subintervals.
constexpr double kCoshLimit = 100.0;  // func_expdisk3d.cpp:64
constexpr double kTinyLog2 = -900.0;

struct LosPixel {
  const CompF64 *c;
  double x_d0, y_d0, z_d0;
};

__device__ __noinline__ double expdisk_ref64(const LosPixel &p, double s) {
  const CompF64 &c = *p.c;
  const double y_d = p.y_d0 + s * c.f;
  const double z = fabs(p.z_d0 - s * c.e);
  const double R = sqrt(p.x_d0 * p.x_d0 + y_d * y_d);
  double vs;
  if ((z / c.h) > kCoshLimit) {
    vs = c.i * exp(-z / c.d);
  } else {
    const double sech = 1.0 / cosh(z / c.h);
    vs = pow(sech, c.g);
  }
  return c.a * exp(-R / c.b) * vs;
}

__device__ __noinline__ double ferrers_ref64(const LosPixel &p, double s) {
  const CompF64 &c = *p.c;
  const double y_d = p.y_d0 + s * c.f;
  const double z_d = p.z_d0 - s * c.e;
  const double x_bar = p.x_d0 * c.g + y_d * c.h;
  const double y_bar = -p.x_d0 * c.h + y_d * c.g;
  const double z_bar = fabs(z_d);
  const double m2 = y_bar * y_bar / c.i + x_bar * x_bar / c.j + z_bar * z_bar / c.k;
  if (m2 > 1.0) return 0.0;
  return c.a * pow((1.0 - m2), c.l);
}

// LuminosityDensity of ExponentialDisk3D along the line of sight s:
//   J_0 exp(-R/h) sech^alpha(|z| / (alpha z_0)),  sech u = 2 e^-u / (1 + e^-2u)
//   = J_0 2^alpha 2^-(R log2 e / h + |z| log2 e / z_0 + alpha log2(1 + e^-2u)).
// (The reference switches to the asymptote 2^alpha e^(-|z|/z_0) beyond u = 100,
// where the last term is below 1e-87.)
struct ExpDiskLos64 {
  const Fp64Tables *t;
  LosPixel p;
  double x2, cosInc, sinInc, amp, kR, kz, ku, alpha;
  __device__ double operator()(double s) const {
    const double y_d = fma(s, sinInc, p.y_d0);
    const double z = fabs(fma(-s, cosInc, p.z_d0));
    const double R2 = fma(y_d, y_d, x2);
    const double R = __double2hiint(R2) >= 0x20000000 ? sqrt64(R2) : 0.0;  // (below 1e-154: 0)
    const double arg = fma(R, kR, z * kz);
    if (!(arg > kTinyLog2)) return expdisk_ref64(p, s);
    const double e = exp2_hl<true>(*t, z * ku, 0.0);
    const hl64 L = log2_hl(*t, 1.0 + e);
    return amp * exp2_hl<false>(*t, arg, alpha * (L.h + L.l));
  }
};

// LuminosityDensity of FerrersBar3D (the reference pairs y_bar with a^2 and
// x_bar with b^2).  An index of 1, 2 or 3 multiplies, others go through
// 2^(n log2(1 - m^2)).
struct FerrersLos64 {
  const Fp64Tables *t;
  LosPixel p;
  double xc, xs, cosInc, sinInc, cosB, sinB, J_0, ia2, ib2, ic2, n;
  __device__ double operator()(double s) const {
    const double y_d = fma(s, sinInc, p.y_d0);
    const double z_d = fma(-s, cosInc, p.z_d0);
    const double x_bar = fma(y_d, sinB, xc);
    const double y_bar = fma(y_d, cosB, -xs);
    const double w = 1.0 - fma(y_bar * y_bar, ia2, fma(x_bar * x_bar, ib2, z_d * z_d * ic2));
    if (w < 0.0) return 0.0;
    if (n == 2.0) return J_0 * (w * w);
    if (n == 1.0) return J_0 * w;
    if (n == 3.0) return J_0 * (w * w * w);
    if (__double2hiint(w) < 0x20000000) return ferrers_ref64(p, s);
    const hl64 L = scale_hl(log2_hl(*t, w), n);
    if (!(L.h > kTinyLog2)) return ferrers_ref64(p, s);
    return J_0 * exp2_hl<false>(*t, L.h, L.l);
  }
};

// The reference's expressions throughout: an integral that the forms above
// cannot bring below the device's 64 subintervals is tried again with these,
// so that exactly the integrals that need more with the reference's rounding
// are refused.
struct RefLos64 {
  LosPixel p;
  __device__ double operator()(double s) const {
    return p.c->type == F_EXPDISK3D ? expdisk_ref64(p, s) : ferrers_ref64(p, s);
  }
};
__device__ __noinline__ int los_retry64(const LosPixel &p, double lim, double &result) {
  return qags_integrate(RefLos64{p}, -lim, lim, kLosEpsRel, result);
}

// GetValue(x, y) of a 3-D component (FP64 fields as comp_setup64 fills them).
__device__ double los_value64(const Fp64Tables &tab, const CompF64 &c, double x, double y, int &status) {
  double x_diff = x - c.x0, y_diff = y - c.y0;
  double xp = x_diff * c.cosPA + y_diff * c.sinPA;
  double yp = -x_diff * c.sinPA + y_diff * c.cosPA;
  double result = 0.0;
  const LosPixel p{&c, xp, yp * c.e, yp * c.f};
  if (c.type == F_EXPDISK3D) {
    ExpDiskLos64 f;
    f.t = &tab;
    f.p = p;
    f.x2 = xp * xp;
    f.cosInc = c.e;
    f.sinInc = c.f;
    f.amp = c.a * c.i;
    f.kR = -kLog2e64 / c.b;
    f.kz = -kLog2e64 / c.d;
    f.ku = -2.0 * kLog2e64 / c.h;
    f.alpha = -c.g;
    const double lim = kExpDiskIntegMult * c.b;
    status = qags_integrate(f, -lim, lim, kLosEpsRel, result);
    if (status == kQagsCapped) status = los_retry64(p, lim, result);
  } else {
    FerrersLos64 f;
    f.t = &tab;
    f.p = p;
    f.xc = xp * c.g;
    f.xs = xp * c.h;
    f.cosInc = c.e;
    f.sinInc = c.f;
    f.cosB = c.g;
    f.sinB = c.h;
    f.J_0 = c.a;
    f.ia2 = 1.0 / c.i;
    f.ib2 = 1.0 / c.j;
    f.ic2 = 1.0 / c.k;
    f.n = c.l;
    const double lim = c.m;
    status = qags_integrate(f, -lim, lim, kLosEpsRel, result);
    if (status == kQagsCapped) status = los_retry64(p, lim, result);
  }
  return result;
}

// out[k3 * n + pixel]: value of the k3-th 3-D component at every model pixel.
// Pixel coordinates as in k_eval64.  *flag gets bit 0 set when an integral
// needed more subintervals than the device list holds.
__global__ void __launch_bounds__(128) k_los64(const CompF64 *__restrict__ comps, LosList64 list,
                                               double *__restrict__ out, Grid64 g, int *__restrict__ flag) {
  __shared__ Fp64Tables tab;
  fp64_tables_load(tab);
  __syncthreads();
  const long n = (long)g.nCols * g.nRows;
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const CompF64 &c = comps[list.comp[blockIdx.y]];
  const long j = k % g.nCols, i = k / g.nCols;
  double x, y;
  if (!g.isRegion) {
    y = (double)(i - g.pr + 1);
    x = (double)(j - g.pc + 1);
  } else {
    y = g.y1 + g.off + (i - g.pr) * g.frac;
    x = g.x1 + g.off + (j - g.pc) * g.frac;
  }
  int status = 0;
  out[(long)blockIdx.y * n + k] = los_value64(tab, c, x, y, status);
  if (status == kQagsCapped) atomicOr(flag, 1);
}

cudaError_t launch_los64(const CompF64 *comps, const LosList64 &list, double *out, Grid64 g, int *flag,
                         cudaStream_t st) {
  const long n = (long)g.nCols * g.nRows;
  if (n == 0 || list.n == 0) return cudaSuccess;
  k_los64<<<dim3((unsigned)((n + 127) / 128), list.n), 128, 0, st>>>(comps, list, out, g, flag);
  return cudaGetLastError();
}

}  // namespace imfit

namespace imfit {

// FindTotalFluxes' grid integration (core/model_object.cpp:2415-2470): the sum
// of one component's GetValue over an xSize x ySize image with IRAF pixel
// centres (x = j+1, y = i+1).  Grid-stride over pixels, one FP64 partial per
// block (tree reduction in a fixed order); the host adds the partials.
__global__ void __launch_bounds__(256) k_flux64(CompF64 c, int xSize, int ySize, double *__restrict__ partials,
                                                int *__restrict__ flag) {
  __shared__ double red[256];
  __shared__ Fp64Tables tab;
  fp64_tables_load(tab);
  __syncthreads();
  const long n = (long)xSize * ySize;
  double acc = 0.0;
  for (long k = blockIdx.x * (long)blockDim.x + threadIdx.x; k < n; k += (long)gridDim.x * blockDim.x) {
    const long i = k / xSize, j = k - i * xSize;
    const double x = (double)(j + 1), y = (double)(i + 1);
    if (c.type == F_EXPDISK3D || c.type == F_FERRERS3D) {
      int status = 0;
      acc += los_value64(tab, c, x, y, status);
      if (status == kQagsCapped) atomicOr(flag, 1);
    } else {
      acc += comp_value64_2d(c, x, y);
    }
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) partials[blockIdx.x] = red[0];
}

cudaError_t launch_flux64(const CompF64 &c, int xSize, int ySize, double *partials, int nBlocks, int *flag,
                          cudaStream_t st) {
  k_flux64<<<nBlocks, 256, 0, st>>>(c, xSize, ySize, partials, flag);
  return cudaGetLastError();
}

}  // namespace imfit
