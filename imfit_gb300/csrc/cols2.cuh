// cols2.cuh -- one column group of the FP32 convolution in two register
// passes (k_cols2.cu: the launch and what it measures).
#pragma once
#include "kernels.h"

namespace imfit {

namespace {

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
struct ColJob {
  cplx<float> *spec;     // first row, this thread's column
  const cplx<float> *H;  // first row, this thread's column
  int pitch, hPitch;
  int nRowsIn, nRowsOut;
  int R1, R2, P;
  float scale, conj;  // conj: +-scale, the sign of the PSF spectrum's imaginary part
  int cpb;
  bool valid;         // the column exists (others read the last one and write nothing)
};

// This thread's share of the twiddle table has arrived; then everyone's.  A
// barrier of the CTA that whole warps reach here or in cols_first.
__device__ __forceinline__ void twiddles_ready() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\nbar.sync 0;\n" ::: "memory");
}

// Called by whole warps (it holds the barrier); the threads with t < R2 have
// work.
template <int R1>
__device__ __noinline__ void cols_first(const ColJob &jr, int t, cplx<float> *sm, const cplx<float> *tw) {
  const ColJob j = jr;  // in registers: a reference would be re-read after every store
  const int n2 = min(t, j.R2 - 1);
  cplx<float> v[R1];
  const cplx<float> *src = j.spec;
  int row = n2;
#pragma unroll
  for (int n1 = 0; n1 < R1; n1++) {
    v[n1] = row < j.nRowsIn ? src[row * j.pitch] : cplx<float>{0.f, 0.f};
    row += j.R2;
  }
  dft_reg<R1, -1>(v);
  twiddles_ready();
  if (t >= j.R2) return;
  int o = n2;
#pragma unroll
  for (int k1 = 0; k1 < R1; k1++) {
    sm[o * j.cpb] = k1 ? cmul(v[k1], tw[o]) : v[0];
    o += j.P;
  }
}

template <int R2>
__device__ __noinline__ void cols_mid(const ColJob &jr, int k1, cplx<float> *sm, const cplx<float> *tw) {
  const ColJob j = jr;
  cplx<float> v[R2];
  cplx<float> *d = sm + k1 * j.P * j.cpb;
#pragma unroll
  for (int n2 = 0; n2 < R2; n2++) v[n2] = d[n2 * j.cpb];
  dft_reg<R2, -1>(v);
  int row = k1;
#pragma unroll
  for (int k2 = 0; k2 < R2; k2++) {
    cplx<float> w = j.H[row * j.hPitch];
    row += j.R1;
    w.x *= j.scale;
    w.y *= j.conj;
    v[k2] = cmul(v[k2], w);
  }
  dft_reg<R2, 1>(v);
  tw += k1 * j.P;
#pragma unroll
  for (int n2 = 0; n2 < R2; n2++) {
    cplx<float> w = tw[n2];
    w.y = -w.y;
    d[n2 * j.cpb] = n2 ? cmul(v[n2], w) : v[0];
  }
}

template <int R1>
__device__ __noinline__ void cols_last(const ColJob &jr, int n2, const cplx<float> *sm) {
  const ColJob j = jr;
  cplx<float> v[R1];
  int o = n2;
#pragma unroll
  for (int k1 = 0; k1 < R1; k1++) {
    v[k1] = sm[o * j.cpb];
    o += j.P;
  }
  dft_reg<R1, 1>(v);
  if (!j.valid) return;
  int row = n2;
#pragma unroll
  for (int n1 = 0; n1 < R1; n1++) {
    if (row < j.nRowsOut) j.spec[row * j.pitch] = v[n1];
    row += j.R2;
  }
}

// spec and H point at the CTA's first column; nl columns exist
__device__ __forceinline__ void cols_two_pass(unsigned char *smem_raw, cplx<float> *spec, long pitch, int nl,
                                              int nRowsIn, int nRowsOut, const cplx<float> *H, long hPitch,
                                              const TwoPass &f, float scale, float conj, int cpb) {
  const int P = two_pass_pitch(f.R2), nT = two_pass_table(f.R1, f.R2);
  cplx<float> *tw = reinterpret_cast<cplx<float> *>(smem_raw);
  cplx<float> *sm = tw + nT;
  // twiddles on their way while the first pass loads and runs
  for (int i = threadIdx.x; 2 * i < nT; i += blockDim.x) cp_async16(tw + 2 * i, f.t + 2 * i);
  const int l = threadIdx.x & (cpb - 1), t = threadIdx.x / cpb;
  const int lc = min(l, nl - 1);
  const ColJob j{spec + lc, H + lc, (int)pitch, (int)hPitch, nRowsIn, nRowsOut, f.R1, f.R2, P, scale, conj, cpb, l < nl};
  sm += l;
  if ((int)(threadIdx.x & ~31u) < f.R2 * cpb) {
    switch (f.R1) {
#define X(R) case R: cols_first<R>(j, t, sm, tw); break;
      IMFIT_TWO_PASS_RADICES(X)
#undef X
    }
  } else {
    twiddles_ready();
  }
  __syncthreads();
  if (t < f.R1) {
    switch (f.R2) {
#define X(R) case R: cols_mid<R>(j, t, sm, tw); break;
      IMFIT_TWO_PASS_RADICES(X)
#undef X
    }
  }
  __syncthreads();
  pdl_trigger();
  if (t < f.R2) {
    switch (f.R1) {
#define X(R) case R: cols_last<R>(j, t, sm); break;
      IMFIT_TWO_PASS_RADICES(X)
#undef X
    }
  }
}

}  // namespace

}  // namespace imfit
