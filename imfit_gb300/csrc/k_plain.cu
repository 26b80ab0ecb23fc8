// k_plain.cu -- the plain FP64 path: the drop-in for ModelObject's
// CreateModelImage / ComputeDeviates / GetFitStatistic.
//
// Compiled with --fmad=false: every expression is evaluated in the same order
// and with the same rounding as the reference's (non-FMA) x86 build, so the
// per-pixel model matches ModelObject::CreateModelImage to a few ulp (the
// transcendental functions are CUDA's, not glibc's).
#include <algorithm>

#include "fp64_math.cuh"
#include "kernels.h"
#include "stat_common.cuh"

namespace imfit {

// Coordinates of model pixel (i, j): IRAF pixel centres on the main grid,
// subpixel centres on a region grid.
__device__ __forceinline__ void pixel_xy64(const Grid64 &g, long i, long j, double &x, double &y) {
  if (!g.isRegion) {
    y = (double)(i - g.pr + 1);
    x = (double)(j - g.pc + 1);
  } else {
    y = g.y1 + g.off + (i - g.pr) * g.frac;
    x = g.x1 + g.off + (j - g.pc) * g.frac;
  }
}

// classes with a subsampling rule (n_subsamples64)
__device__ __forceinline__ bool subsampled64(int t) {
  return t == F_SERSIC || t == F_EXP || t == F_MOFFAT || t == F_GAUSS;
}

// Subsample count at (x, y), with comp_value64_2d's expressions.
__device__ __forceinline__ int n_subsamples_at64(const CompF64 &c, double x, double y) {
  const double x_diff = x - c.x0, y_diff = y - c.y0;
  const double xp = x_diff * c.cosPA + y_diff * c.sinPA;
  const double yps = (-x_diff * c.sinPA + y_diff * c.cosPA) / c.q;
  return n_subsamples64(c, sqrt(xp * xp + yps * yps));
}

// Box of 2 subHalf x 2 subHalf pixels around component c's centre: every
// pixel within radius 10 of it (the only ones the subsampling rules touch)
// lies inside.  Origin (j0, i0).
__device__ __forceinline__ void sub_box64(const Grid64 &g, const CompF64 &c, long &j0, long &i0) {
  double jc, ic;
  if (!g.isRegion) {
    jc = c.x0 + g.pc - 1;
    ic = c.y0 + g.pr - 1;
  } else {
    jc = (c.x0 - g.x1 - g.off) / g.frac + g.pc;
    ic = (c.y0 - g.y1 - g.off) / g.frac + g.pr;
  }
  j0 = (long)floor(jc) - g.subHalf + 1;
  i0 = (long)floor(ic) - g.subHalf + 1;
}

size_t sub_table_size(const Grid64 &g, int nComp) {
  const long S = 2L * g.subHalf;
  return (size_t)nComp * S * S;
}

// r (h + l) as an unevaluated sum
__device__ __forceinline__ hl64 times_hl(double r, double h, double l) {
  const double p = r * h;
  return {p, fma(r, l, fma(r, h, -p))};
}

// Squared radius of a pixel at offsets dx, dy from a component's centre
// (comp_fast64's form: one multiplication by 1/q instead of a division).
__device__ __forceinline__ double radius2_fast64(const CompF64 &c, double dx, double dy) {
  const double xp = fma(dx, c.cosPA, dy * c.sinPA);
  const double yp = fma(dy, c.cosPA, -dx * c.sinPA);
  const double ys = fma(yp, c.iqh, yp * c.iql);
  return fma(xp, xp, ys * ys);
}

// Profile of a radial class at squared radius v (normal and finite) with
// comp_fast64's constants: 38 FP64 instructions (Sersic), 20 (Exponential),
// 14 (Gaussian) instead of 190, 40 and 30 with the library's pow and exp,
// divisions and square root.
__device__ __forceinline__ double radial_fast64(const Fp64Tables &t, const CompF64 &c, double v) {
  switch (c.type) {
    case F_SERSIC: {  // I_e 2^(B (1 - 2^(log2((r/r_e)^2) / 2n)))
      hl64 L = log2_hl(t, v);
      L.h -= c.vh;
      L.l -= c.vl;
      const hl64 e = scale_hl(L, c.u);
      const double w = 1.0 - exp2_hl<false>(t, e.h, e.l);
      const hl64 a = times_hl(w, c.uh, c.ul);
      return c.b * exp2_hl<true>(t, a.h, a.l);
    }
    case F_EXP: {
      const hl64 a = times_hl(-sqrt64(v), c.uh, c.ul);
      return c.a * exp2_hl<true>(t, a.h, a.l);
    }
    case F_GRING: {
      const double d = sqrt64(v) - c.b;
      const hl64 a = times_hl(-(d * d), c.uh, c.ul);
      return c.a * exp2_hl<true>(t, a.h, a.l);
    }
    case F_MOFFAT: {
      const hl64 e = scale_hl(log2_hl(t, 1.0 + fma(v, c.uh, v * c.ul)), c.u);
      return c.a * exp2_hl<false>(t, e.h, e.l);
    }
    default: {  // F_GAUSS
      const hl64 a = times_hl(-v, c.uh, c.ul);
      return c.a * exp2_hl<true>(t, a.h, a.l);
    }
  }
}

// A subsample of a pixel: any radius, the centre included.
__device__ __forceinline__ double radial_sub64(const Fp64Tables &t, const CompF64 &c, double xi, double yi) {
  const double dx = xi - c.x0, dy = yi - c.y0;
  const double v = radius2_fast64(c, dx, dy);
  if (c.farHi != 0x7fffffff && __double2hiint(v) >= 0x20000000) return radial_fast64(t, c, v);
  const double xp = dx * c.cosPA + dy * c.sinPA;
  const double yps = (-dx * c.sinPA + dy * c.cosPA) / c.q;
  return radial64(c, sqrt(xp * xp + yps * yps));
}

// ---- subsampled pixels -----------------------------------------------------
// The subsampled pixels of a component (within radius 10 of its centre, at
// most 100 x 100 subsamples each; 400 inside the constant-count radius) go
// into a table over a box around the centre.  The work is FP64-throughput
// bound and very uneven over the box, so it is spread over the whole GPU and
// over the lanes: a CTA takes box pixels that lie gridDim.x apart, every
// thread classifies one, and a pixel of n x n subsamples is then summed by 4
// lanes (n = 2), 16 (n = 3, 4), a warp (up to kSubWarp subsamples) or the whole
// CTA, which evaluates the terms into shared memory.  Measured: main grid of a
// 256 x 256 Sersic 104 us with one warp per pixel on adjacent pixels (the 50
// central pixels' 25,000 evaluations on ten SMs), 5x region 417 us.
//
// The order of a sum does not depend on the split: lane l of one warp adds
// subsamples l, l + 32, ... in sequence, then a fixed tree (fewer lanes leave
// out only zeros) -- different from the reference's single sequence by FP64
// rounding only (~1e-16 relative).
constexpr int kSubWarp = 64;

// the shared subsample lattice of an oversampled region (lattice form below)
struct Lattice64 {
  double *val;    // [vector][component][side * side], or null
  int q0, count;  // box pixels [q0, q0 + count) use it
  int step;       // lattice points per box pixel
  int side;
};
constexpr int kLattice = 20;  // subsamples per axis of the constant-count rule

__device__ __forceinline__ bool sub_changed(const unsigned *changed, int vec, int c) {
  return !changed || (changed[vec] >> c) & 1u;
}

// Lattice of a region of scale k, 20 % k == 0: the subsamples of its pixels
// span a whole main pixel, so those of neighbouring pixels coincide; every
// pixel with the constant 20 x 20 count (radius 4) sums a 20 x 20 block of one
// lattice of spacing 1/20, 20/k points further per pixel.  One thread per
// point: 34,000 evaluations a component at k = 5 instead of 630,000.
__global__ void __launch_bounds__(128) k_lattice64(const CompF64 *__restrict__ comps, int nComp, Grid64 g,
                                                   Lattice64 L, const unsigned *__restrict__ changed) {
  __shared__ Fp64Tables tab;
  const int c = blockIdx.y, vec = blockIdx.z;
  const CompF64 cc = comps[(long)vec * nComp + c];
  if (!cc.subsample || !subsampled64(cc.type) || !sub_changed(changed, vec, c)) return;
  fp64_tables_load(tab);
  __syncthreads();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= L.side * L.side) return;
  long j0, i0;
  sub_box64(g, cc, j0, i0);
  double x, y;
  pixel_xy64(g, i0 + L.q0, j0 + L.q0, x, y);
  const double d = 1.0 / kLattice;
  const int r = p / L.side, a = p - r * L.side;
  L.val[((long)vec * nComp + c) * L.side * L.side + p] =
      radial_sub64(tab, cc, (x - 0.5 + 0.5 * d) + a * d, (y - 0.5 + 0.5 * d) + r * d);
}

// Box pixels of one CTA: at most 256, so that each thread classifies one.
constexpr int kSubPixels = 64;

__global__ void __launch_bounds__(256) k_sub64(const CompF64 *__restrict__ comps, int nComp, Grid64 g, Lattice64 L,
                                               const unsigned *__restrict__ changed) {
  constexpr int kChunk = 1024;
  __shared__ Fp64Tables tab;
  __shared__ short pix[4][kSubPixels], num[4][kSubPixels];  // by class: index in the CTA's pixels, n
  __shared__ int cnt[4];
  __shared__ double term[kChunk];
  const int c = blockIdx.y, vec = blockIdx.z;
  const CompF64 &cc = comps[(long)vec * nComp + c];
  if (!cc.subsample || !subsampled64(cc.type) || !sub_changed(changed, vec, c)) return;
  const int S = 2 * g.subHalf, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  long j0, i0;
  sub_box64(g, cc, j0, i0);
  // coordinates of the CTA's pixel e, and its box index
  auto place = [&](int e, double &x, double &y) {
    const int p = (int)blockIdx.x + e * (int)gridDim.x;
    pixel_xy64(g, i0 + p / S, j0 + p % S, x, y);
    return p;
  };
  if (threadIdx.x < 4) cnt[threadIdx.x] = 0;
  __syncthreads();
  int mine = 1;
  if (threadIdx.x < kSubPixels) {
    const int e = threadIdx.x, p = (int)blockIdx.x + e * (int)gridDim.x;
    const long i = i0 + p / S, j = j0 + p % S;
    if (p < S * S && i >= 0 && i < g.nRows && j >= 0 && j < g.nCols) {
      double x, y;
      place(e, x, y);
      mine = n_subsamples_at64(cc, x, y);
    }
    if (mine > 1) {
      const int br = p / S, bc = p - br * S;
      const bool lat =
          L.val && mine == kLattice && br >= L.q0 && br < L.q0 + L.count && bc >= L.q0 && bc < L.q0 + L.count;
      const int k = mine == 2 ? 0 : (mine <= 4 ? 1 : ((lat || mine * mine <= kSubWarp) ? 2 : 3));
      const int at = atomicAdd(&cnt[k], 1);
      pix[k][at] = (short)e;
      num[k][at] = (short)(lat ? -mine : mine);
    }
  }
  if (!__syncthreads_or(mine > 1)) return;
  fp64_tables_load(tab);
  __syncthreads();
  double *out = g.sub + ((long)vec * nComp + c) * S * S;
  // subsample t of the n x n of the pixel at (xx, yy)
  auto value = [&](double xx, double yy, int n, int t) {
    const double d = 1.0 / n;
    const double xs0 = xx - 0.5 + 0.5 * d;
    const double ys0 = yy - 0.5 + 0.5 * d;
    const int ii = t / n, jj = t - ii * n;
    return radial_sub64(tab, cc, xs0 + ii * d, ys0 + jj * d);
  };
  auto tree = [](double s, int group) {
    for (int o = group / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
  };
  for (int k = 0; k < 3; k++) {
    const int group = k == 0 ? 4 : (k == 1 ? 16 : 32), per = 32 / group, gl = lane & (group - 1);
    for (int e0 = wid * per; e0 < cnt[k]; e0 += 8 * per) {  // uniform over the warp
      const int e = e0 + lane / group;
      int n = 0, p = 0;
      double x = 0.0, y = 0.0, s = 0.0;
      if (e < cnt[k]) {
        n = num[k][e];
        p = place(pix[k][e], x, y);
      }
      if (n < 0) {  // on the lattice (k = 2): lane i adds column i of its block
        const int br = p / S, bc = p - br * S;
        const double *b = L.val + ((long)vec * nComp + c) * L.side * L.side +
                          (long)(br - L.q0) * L.step * L.side + (bc - L.q0) * L.step + lane;
        if (lane < kLattice)
#pragma unroll
          for (int r = 0; r < kLattice; r++) s += b[(long)r * L.side];
      } else {
        for (int t = gl; t < n * n; t += group) s += value(x, y, n, t);
      }
      s = tree(s, group);
      if (gl == 0 && n) out[p] = s / (n * n);
    }
  }
  for (int e = 0; e < cnt[3]; e++) {
    const int n = num[3][e];
    double x, y, s = 0.0;
    const int p = place(pix[3][e], x, y);
    for (int t0 = 0; t0 < n * n; t0 += kChunk) {
      const int m = min(kChunk, n * n - t0);
      for (int t = threadIdx.x; t < m; t += 256) term[t] = value(x, y, n, t0 + t);
      __syncthreads();
      if (wid == 0)
        for (int t = lane; t < m; t += 32) s += term[t];
      __syncthreads();
    }
    if (wid == 0) {
      s = tree(s, 32);
      if (lane == 0) out[p] = s / (n * n);
    }
  }
}

// CreateModelImage pixel loop: core/model_object.cpp:1144-1175 (main grid),
// OversampledRegion::ComputeRegionAndDownsample core/oversampled_region.cpp:301-327
// (region grid).  One thread per model pixel; Kahan sum over components in
// their order; subsampled pixels from k_sub64's table, the others outside
// radius 10 by the few-instruction form.
//
// FP64-issue bound.  A Sersic + Exponential + FlatSky pixel takes about 100
// FP64 instructions instead of 242.
//
// Several parameter vectors at once (MODE): kOne, one vector; kBase, also
// store each component's values to base[c][pixel]; kDelta, vector 1 +
// blockIdx.z: components that differ from vector 0's (changed bit c) are
// evaluated, the others' values read from base -- a finite-difference step
// changes the components of one function set at most, so a gradient of P
// parameters costs about P component images, not P x components.
enum EvalMode { kOne = 0, kBase = 1, kDelta = 2 };

template <int MODE>
__global__ void __launch_bounds__(128) k_eval64(const CompF64 *__restrict__ comps, int nComp,
                                                double *__restrict__ model, long pitch, long modelStride, Grid64 g,
                                                const double *__restrict__ los, double *__restrict__ base,
                                                const unsigned *__restrict__ changed) {
  __shared__ CompF64 sc[kMaxComponents];
  __shared__ Fp64Tables tab;
  const int vec = MODE == kDelta ? 1 + blockIdx.z : 0;
  {
    const int n = nComp * (int)(sizeof(CompF64) / sizeof(double));
    const double *src = reinterpret_cast<const double *>(comps + (long)vec * nComp);
    double *dst = reinterpret_cast<double *>(sc);
    for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
  }
  fp64_tables_load(tab);
  __syncthreads();
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= g.nCols) return;
  const unsigned ch = MODE == kDelta ? changed[vec] : 0xffffffffu;
  const long n = (long)g.nCols * g.nRows;
  const int S = 2 * g.subHalf;
  for (int i = blockIdx.y; i < g.nRows; i += gridDim.y) {
    const long k = (long)i * g.nCols + j;
    double x, y;
    pixel_xy64(g, i, j, x, y);
    double s = 0.0, err = 0.0;
    for (int c = 0; c < nComp; c++) {
      const CompF64 &cc = sc[c];
      const int t = cc.type;
      if (is_point_source(t)) continue;  // added after the convolution
      double v;
      if (t == F_FLATSKY || t == F_TILTEDSKY) {
        v = comp_value64_2d(cc, x, y);
      } else if (MODE == kDelta && !((ch >> c) & 1u)) {
        v = base[c * n + k];
      } else if (t == F_EXPDISK3D || t == F_FERRERS3D) {
        v = los[(long)cc.pad0 * n + k];
      } else {
        const double dx = x - cc.x0, dy = y - cc.y0;
        const double r2 = radius2_fast64(cc, dx, dy);
        if (__double2hiint(r2) >= cc.farHi) {
          v = radial_fast64(tab, cc, r2);
        } else {
          // comp_value64_2d with the subsampled pixels read from the table
          const double xp = dx * cc.cosPA + dy * cc.sinPA;
          const double yps = (-dx * cc.sinPA + dy * cc.cosPA) / cc.q;
          const double r = sqrt(xp * xp + yps * yps);
          if (n_subsamples64(cc, r) > 1) {
            long j0, i0;
            sub_box64(g, cc, j0, i0);
            const long bi = i - i0, bj = j - j0;
            v = (bi >= 0 && bi < S && bj >= 0 && bj < S) ? g.sub[((long)vec * nComp + c) * S * S + bi * S + bj]
                                                         : comp_value64_2d(cc, x, y);
          } else {
            v = radial64(cc, r);
          }
        }
        if (MODE == kBase) base[c * n + k] = v;
      }
      const double adj = v - err;
      const double tmp = s + adj;
      err = (tmp - s) - adj;
      s = tmp;
    }
    model[vec * modelStride + (long)i * pitch + j] = s;
  }
}

size_t lattice_size(const Grid64 &g, int nComp) {
  if (!g.isRegion || g.scale < 1 || kLattice % g.scale) return 0;
  const size_t side = (size_t)(8 * g.scale + 1) * (kLattice / g.scale) + kLattice;
  return side * side * nComp;
}

// comps: nVec vectors of nComp components; with nVec > 1, base (nComp values
// per pixel) and changed (nVec masks on the device) describe vectors 1.. as
// differences from vector 0.
cudaError_t launch_eval64(const CompF64 *comps, int nComp, double *model, long pitch, Grid64 g, const double *los,
                          cudaStream_t st, int nVec, long modelStride, double *base, const unsigned *changed) {
  if (g.nCols <= 0 || g.nRows <= 0) return cudaSuccess;
  const int S = 2 * g.subHalf;
  Lattice64 L{};
  if (g.lattice && lattice_size(g, 1)) {
    L.val = g.lattice;
    L.q0 = g.subHalf - 1 - 4 * g.scale;  // box pixels within radius 4 of the centre
    L.count = 8 * g.scale + 2;
    L.step = kLattice / g.scale;
    L.side = (L.count - 1) * L.step + kLattice;
    k_lattice64<<<dim3((unsigned)((L.side * L.side + 127) / 128), nComp, nVec), 128, 0, st>>>(comps, nComp, g, L,
                                                                                             changed);
  }
  // main grid: four box pixels per CTA, so that the few large ones are spread
  // as widely as they can be; region: its many small ones fill the lanes
  const int per = g.isRegion ? kSubPixels : 4;
  k_sub64<<<dim3((unsigned)((S * S + per - 1) / per), nComp, nVec), 256, 0, st>>>(comps, nComp, g, L, changed);
  // a row of pixels per CTA row; narrow grids take narrower CTAs
  const int threads = g.nCols >= 128 ? 128 : std::max(32, (g.nCols + 31) / 32 * 32);
  const dim3 grid((g.nCols + threads - 1) / threads, std::min(g.nRows, 65535));
  if (nVec == 1) {
    k_eval64<kOne><<<grid, threads, 0, st>>>(comps, nComp, model, pitch, modelStride, g, los, nullptr, nullptr);
  } else {
    k_eval64<kBase><<<grid, threads, 0, st>>>(comps, nComp, model, pitch, modelStride, g, los, base, nullptr);
    k_eval64<kDelta><<<dim3(grid.x, grid.y, nVec - 1), threads, 0, st>>>(comps, nComp, model, pitch, modelStride, g,
                                                                        los, base, changed);
  }
  return cudaGetLastError();
}

// Point sources after the convolution: core/model_object.cpp:1183-1216 on the
// main grid, core/oversampled_region.cpp:363-408 on a region grid.  Kahan sum
// over the point sources, added to the model.  Value I_tot * P(s (x - x0),
// s (y - y0)) (func_pointsource.cpp:220-229), rotated by PA for PointSourceRot
// (func_pointsource-rot.cpp:229-243); s = scales.s[c], the component's
// PointSource::oversamplingScale for this pass.
__global__ void __launch_bounds__(256) k_point_sources64(const CompF64 *__restrict__ comps, int nComp,
                                                         double *__restrict__ model, long pitch, Grid64 g,
                                                         PsfInterp<double> ip, PsScales scales) {
  __shared__ CompF64 sc[kMaxComponents];
  for (int i = threadIdx.x; i < nComp; i += blockDim.x) sc[i] = comps[i];
  __syncthreads();
  const long n = (long)g.nCols * g.nRows;
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const long j = k % g.nCols, i = k / g.nCols;
  double x, y;
  if (!g.isRegion) {
    y = (double)(i - g.pr + 1);
    x = (double)(j - g.pc + 1);
  } else {
    y = g.y1 + g.off + (i - g.pr) * g.frac;
    x = g.x1 + g.off + (j - g.pc) * g.frac;
  }
  double s = 0.0, err = 0.0;
  for (int c = 0; c < nComp; c++) {
    const CompF64 &f = sc[c];
    if (!is_point_source(f.type)) continue;
    const double os = (double)scales.s[c];
    double xd = os * (x - f.x0), yd = os * (y - f.y0);
    if (f.type == F_POINTSOURCEROT) {
      const double xp = xd * f.cosPA + yd * f.sinPA;
      const double yp = -xd * f.sinPA + yd * f.cosPA;
      xd = xp;
      yd = yp;
    }
    const double v = f.a * psf_interp64(ip, xd, yd);
    const double adj = v - err;
    const double tmp = s + adj;
    err = (tmp - s) - adj;
    s = tmp;
  }
  model[i * pitch + j] += s;
}

cudaError_t launch_point_sources64(const CompF64 *comps, int nComp, double *model, long pitch, Grid64 g,
                                   PsfInterp<double> ip, const PsScales &scales, cudaStream_t st) {
  const long n = (long)g.nCols * g.nRows;
  if (n == 0) return cudaSuccess;
  k_point_sources64<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(comps, nComp, model, pitch, g, ip, scales);
  return cudaGetLastError();
}

// DownsampleAndReplace: core/downsample.cpp:54-109, over the nColsSub x
// nRowsSub data pixels it replaces (the caller applies its size rule); the
// region's first subpixel lies at (padR, padC) of its model grid.
__global__ void k_downsample64(const double *__restrict__ os, int nOC, int padC, int padR,
                               double *__restrict__ mainImg, int nMainCols, int i1, int j1, int nColsSub,
                               int nRowsSub, int scale, long osStride, long mainStride) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nColsSub * nRowsSub) return;
  os += blockIdx.y * osStride;
  mainImg += blockIdx.y * mainStride;
  const int i_sub = t / nColsSub, j_sub = t % nColsSub;
  const int jj1 = j_sub * scale + padC;
  const int ii1 = i_sub * scale + padR;
  double b = 0.0;
  for (int ii = ii1; ii < ii1 + scale; ii++)
    for (int jj = jj1; jj < jj1 + scale; jj++) b += os[(long)ii * nOC + jj];
  const double area = scale * scale;
  mainImg[(long)(i1 + i_sub) * nMainCols + (j1 + j_sub)] = b / area;
}

cudaError_t launch_downsample64(const double *region, int nOC, int padC, int padR, int nColsSub, int nRowsSub,
                                double *mainImg, int nMainCols, int mainPsfCols, int mainPsfRows, int x1, int y1,
                                int scale, cudaStream_t st, int nVec, long regionStride, long mainStride) {
  const int j1 = x1 - 1 + mainPsfCols;
  const int i1 = y1 - 1 + mainPsfRows;
  const int n = nColsSub * nRowsSub;
  if (n <= 0) return cudaSuccess;
  k_downsample64<<<dim3((n + 127) / 128, nVec), 128, 0, st>>>(region, nOC, padC, padR, mainImg, nMainCols, i1, j1,
                                                              nColsSub, nRowsSub, scale, regionStride, mainStride);
  return cudaGetLastError();
}

// ------------------------------------------------------------- statistics
#define LOG_SMALL_VALUE 1.0e-25  // core/model_object.cpp:86

struct Term {
  double w, d, m, extra;
  long b;
};

__device__ __forceinline__ long model_index(const StatArgs64 &a, long b) {
  const long row = b / a.nDataCols;
  const long col = b - row * a.nDataCols;
  return (long)a.modelCols * (a.offR + row) + a.offC + col;
}

// weight for term b; UpdateWeightVector (core/model_object.cpp:1345-1381)
// when model-based errors are in use
__device__ __forceinline__ double term_weight(const StatArgs64 &a, long b, double m) {
  if (a.modelErrors && a.mask[b] > 0) {
    const double tf = m + a.sky;
    const double ns = tf / a.effGain + a.rnTerm;
    return 1.0 / sqrt(ns);
  }
  return a.weight[b];
}

// ComputeDeviates (core/model_object.cpp:1413-1496) and
// ComputePoissonMLRDeviate (core/model_object.cpp:1386-1401)
__global__ void k_deviates64(StatArgs64 a, double *__restrict__ dev, double *__restrict__ wOut) {
  const long z = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (z >= a.nz) return;
  const long b = a.boot ? a.boot[z] : z;
  const double m = a.model[model_index(a, b)];
  const double w = term_weight(a, b, m);
  if (wOut && a.modelErrors && !a.boot) wOut[b] = w;
  double r;
  if (a.kind == 2) {
    const double mv = a.effGain * (m + a.sky);
    const double dv = a.effGain * (a.data[b] + a.sky);
    const double lm = (mv <= 0) ? LOG_SMALL_VALUE : log(mv);
    r = sqrt(2.0 * w * fabs(mv - dv * lm + a.extra[b]));
  } else {
    r = w * (a.data[b] - m);
  }
  dev[z] = r;
}

cudaError_t launch_deviates64(const StatArgs64 &a, double *dev, double *wOut, cudaStream_t st) {
  if (a.nz <= 0) return cudaSuccess;
  k_deviates64<<<(unsigned)((a.nz + 255) / 256), 256, 0, st>>>(a, dev, wOut);
  return cudaGetLastError();
}

// ChiSquared (core/model_object.cpp:1633-1689) and CashStatistic (:1703-1775),
// first level: fixed grid, grid-stride terms, per-block partial state;
// blockIdx.y: model image (modelStride apart), its partials after the others'.
//
// Bound by the latency of a thread's loads (14 terms a thread for a 1024 x
// 1024 image): four terms' loads are issued before the first is added, and
// pixel rows come from a 32-bit division.  The terms are added in the same
// order as one by one.
constexpr int kStatUnroll = 4;

__device__ __forceinline__ long model_index32(const StatArgs64 &a, long b) {
  const unsigned row = (unsigned)b / (unsigned)a.nDataCols;
  const unsigned col = (unsigned)b - row * (unsigned)a.nDataCols;
  return (long)a.modelCols * (a.offR + (long)row) + a.offC + col;
}

__global__ void __launch_bounds__(256) k_stat64_partial(StatArgs64 a, double *__restrict__ partials,
                                                        long modelStride) {
  const long stride = (long)gridDim.x * blockDim.x;
  a.model += blockIdx.y * modelStride;
  partials += ((long)blockIdx.y * gridDim.x + blockIdx.x) * 5;
  const long z0 = blockIdx.x * (long)blockDim.x + threadIdx.x;
  Enorm e = {0, 0, 0, 0, 0};
  const double agiant = 1.304e19 / (double)(int)a.nz;
  double s = 0.0;
  for (long zb = z0; zb < a.nz; zb += kStatUnroll * stride) {
    double m[kStatUnroll], d[kStatUnroll], w[kStatUnroll], ex[kStatUnroll];
#pragma unroll
    for (int u = 0; u < kStatUnroll; u++) {
      const long z = zb + u * stride;
      m[u] = d[u] = w[u] = ex[u] = 0.0;
      if (z >= a.nz) continue;
      const long b = a.boot ? a.boot[z] : z;
      m[u] = a.model[model_index32(a, b)];
      d[u] = a.data[b];
      w[u] = a.kind == 0 ? term_weight(a, b, m[u]) : a.weight[b];
      if (a.kind != 0) ex[u] = a.extra[b];
    }
#pragma unroll
    for (int u = 0; u < kStatUnroll; u++) {
      if (zb + u * stride >= a.nz) break;
      if (a.kind == 0) {
        enorm_add(e, w[u] * (d[u] - m[u]), agiant);
      } else {
        const double mv = a.effGain * (m[u] + a.sky);
        const double dv = a.effGain * (d[u] + a.sky);
        const double lm = (mv <= 0) ? LOG_SMALL_VALUE : log(mv);
        s += w[u] * (mv - dv * lm + ex[u]);
      }
    }
  }
  if (a.kind == 0) {
    e = block_enorm(e);
    if (threadIdx.x == 0) {
      partials[0] = e.s1; partials[1] = e.x1; partials[2] = e.s2; partials[3] = e.s3; partials[4] = e.x3;
    }
  } else {
    s = block_sum(s);
    if (threadIdx.x == 0) partials[0] = s;
  }
}

__global__ void __launch_bounds__(256) k_stat64_final(const double *__restrict__ partials, int nPart, int kind,
                                                      double *__restrict__ result) {
  partials += (long)blockIdx.x * nPart * 5;
  result += blockIdx.x;
  if (kind == 0) {
    Enorm e = {0, 0, 0, 0, 0};
    for (int i = threadIdx.x; i < nPart; i += blockDim.x) {
      const double *p = partials + i * 5;
      Enorm o = {p[0], p[1], p[2], p[3], p[4]};
      enorm_merge(e, o);
    }
    e = block_enorm(e);
    if (threadIdx.x == 0) {
      const double chi = enorm_final(e);
      *result = chi * chi;
    }
  } else {
    double s = 0.0;
    for (int i = threadIdx.x; i < nPart; i += blockDim.x) s += partials[i * 5];
    s = block_sum(s);
    if (threadIdx.x == 0) *result = 2.0 * s;
  }
}

cudaError_t launch_statistic64(const StatArgs64 &a, double *partials, double *result, cudaStream_t st, int nVec,
                               long modelStride) {
  k_stat64_partial<<<dim3(kStatBlocks, nVec), 256, 0, st>>>(a, partials, modelStride);
  k_stat64_final<<<nVec, 256, 0, st>>>(partials, kStatBlocks, a.kind == 0 ? 0 : 1, result);
  return cudaGetLastError();
}

// Finite-difference column blockIdx.y of the chi^2 gradient: the deviates of
// model 0 and of model 1 + blockIdx.y (ComputeDeviates' expressions), partial
// sums of dev0 (dev1 - dev0) / h.
__global__ void __launch_bounds__(256) k_fd_dot_partial(StatArgs64 a, long modelStride,
                                                        const double *__restrict__ invh,
                                                        double *__restrict__ partials) {
  const long stride = (long)gridDim.x * blockDim.x;
  const double *m1 = a.model + (1 + (long)blockIdx.y) * modelStride;
  const double ih = invh[blockIdx.y];
  double s = 0.0;
  for (long zb = blockIdx.x * (long)blockDim.x + threadIdx.x; zb < a.nz; zb += kStatUnroll * stride) {
    double d0[kStatUnroll], d1[kStatUnroll];
#pragma unroll
    for (int u = 0; u < kStatUnroll; u++) {
      const long z = zb + u * stride;
      d0[u] = d1[u] = 0.0;
      if (z >= a.nz) continue;
      const long b = a.boot ? a.boot[z] : z;
      const long mi = model_index32(a, b);
      const double v0 = a.model[mi], v1 = m1[mi], d = a.data[b];
      d0[u] = term_weight(a, b, v0) * (d - v0);
      d1[u] = term_weight(a, b, v1) * (d - v1);
    }
#pragma unroll
    for (int u = 0; u < kStatUnroll; u++)
      if (zb + u * stride < a.nz) s += d0[u] * ((d1[u] - d0[u]) * ih);
  }
  s = block_sum(s);
  if (threadIdx.x == 0) partials[((long)blockIdx.y * gridDim.x + blockIdx.x) * 5] = s;
}

cudaError_t launch_fd_dot64(const StatArgs64 &a, long modelStride, int nCols, const double *invh, double *partials,
                            double *result, cudaStream_t st) {
  if (nCols <= 0) return cudaSuccess;
  k_fd_dot_partial<<<dim3(kStatBlocks, nCols), 256, 0, st>>>(a, modelStride, invh, partials);
  k_stat64_final<<<nCols, 256, 0, st>>>(partials, kStatBlocks, 1, result);  // returns 2*sum
  return cudaGetLastError();
}

__global__ void k_crop64(const double *__restrict__ model, int modelCols, int offR, int offC, int nCols,
                         int nRows, double *__restrict__ out) {
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (t >= (long)nCols * nRows) return;
  const long r = t / nCols, c = t % nCols;
  out[t] = model[(long)modelCols * (offR + r) + offC + c];
}

cudaError_t launch_crop64(const double *model, int modelCols, int offR, int offC, int nCols, int nRows,
                          double *out, cudaStream_t st) {
  const long n = (long)nCols * nRows;
  if (n == 0) return cudaSuccess;
  k_crop64<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(model, modelCols, offR, offC, nCols, nRows, out);
  return cudaGetLastError();
}

// UpdateWeightVector (core/model_object.cpp:1345-1381): model-based weights
// for unmasked pixels, recomputed after every model image.
__global__ void k_update_weights64(const double *__restrict__ model, const double *__restrict__ mask,
                                   double *__restrict__ weight, long nData, int nDataCols, int modelCols,
                                   int offR, int offC, double effGain, double sky, double rnTerm) {
  const long z = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (z >= nData || !(mask[z] > 0)) return;
  const long row = z / nDataCols, col = z - row * nDataCols;
  const double tf = model[(long)modelCols * (offR + row) + offC + col] + sky;
  const double ns = tf / effGain + rnTerm;
  weight[z] = 1.0 / sqrt(ns);
}

cudaError_t launch_update_weights64(const double *model, const double *mask, double *weight, long nData,
                                    int nDataCols, int modelCols, int offR, int offC, double effGain, double sky,
                                    double rnTerm, cudaStream_t st) {
  if (nData <= 0) return cudaSuccess;
  k_update_weights64<<<(unsigned)((nData + 255) / 256), 256, 0, st>>>(model, mask, weight, nData, nDataCols,
                                                                        modelCols, offR, offC, effGain, sky, rnTerm);
  return cudaGetLastError();
}

__global__ void k_f64_to_f32(const double *__restrict__ in, float *__restrict__ out, long n) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) out[i] = (float)in[i];
}

cudaError_t launch_f64_to_f32(const double *in, float *out, long n, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_f64_to_f32<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(in, out, n);
  return cudaGetLastError();
}

}  // namespace imfit
