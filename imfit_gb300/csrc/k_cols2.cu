// k_cols2.cu -- column pass of the FP32 convolution in two register passes
// (fft2.cuh): the middle step of Convolver::ConvolveImage
// (core/convolver.cpp:365-411) for lengths R1 R2.
//
// A CTA serves cpb adjacent half-spectrum columns (a power of two; thread =
// (n2 or k1, column), columns fastest, so a row's cpb values are one 32- or
// 64-byte piece):
//   1. thread n2 loads its R1 rows straight from the spectrum (all loads in
//      flight at once), transforms, multiplies by W_n^(n2 k1), stores to
//      shared memory;
//   2. thread k1 transforms its R2 values, multiplies by the PSF spectrum
//      (or its conjugate) and 1/(Lx Ly), transforms back, multiplies by the
//      conjugate twiddles, stores in place;
//   3. thread n2 transforms back and stores its rows.
// Half the instructions per point of the multi-pass kernel (k_cols32.cu), but
// long straight-line code at 96 registers: a CTA takes longer, and the kernel
// wins where many share an SM.  Measured (both sides, us): 256 spectra of 576 x
// 289 322 / 333 (291 with packed complex additions), 11 of 1120 x 561 90 / 131,
// 11 of 540 x 271 18 / 31; single spectra lose (1120 x 561 24 / 16, 320 x 161
// 12 / 9), so launch_cols32 takes this form from kTwoPassColumns columns on.
// What it tried and lost: the PSF columns staged in shared memory (two CTAs per
// SM fewer: 404), more CTAs per SM with spilled registers (five: 431).
// Rows at or beyond nRowsIn are implicit zeros, rows from nRowsOut on are not
// written.
#include <algorithm>

#include "cols2.cuh"

namespace imfit {

// Batch entry y uses H + e * hBatch with e = y / hDiv, or hMap[e] when a map
// is given (hBatch 0: one PSF spectrum for every entry).
__global__ void __launch_bounds__(kTwoPassThreads, 4)
    k_cols2(cplx<float> *__restrict__ spec, long pitch, long batch, int nColsC, int nRowsIn, int nRowsOut,
            const cplx<float> *__restrict__ H, long hPitch, TwoPass f, float scale, float conj, int cpb, long hBatch,
            int hDiv, const int *__restrict__ hMap) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_wait();
  if (hBatch) {
    const int e = blockIdx.y / hDiv;
    H += (long)(hMap ? hMap[e] : e) * hBatch;
  }
  const int c0 = blockIdx.x * cpb;
  cols_two_pass(smem_raw, spec + blockIdx.y * batch + c0, pitch, min(cpb, nColsC - c0), nRowsIn, nRowsOut, H + c0,
                hPitch, f, scale, conj, cpb);
}

size_t cols2_smem(const TwoPass &f, int cpb) {
  return sizeof(cplx<float>) * (two_pass_table(f.R1, f.R2) + (size_t)f.R1 * two_pass_pitch(f.R2) * cpb);
}

// columns per CTA: the widest power of two whose threads fit
int cols2_cpb(const TwoPass &f, int most) {
  int c = 1;
  while (c < most && 2 * c * std::max(f.R1, f.R2) <= kTwoPassThreads) c *= 2;
  return c;
}

cudaError_t launch_cols2(void *spec, long pitch, long batch, int nColsC, int nRowsIn, int nRowsOut, const void *H,
                         long hPitch, const TwoPass &f, float scale, int mode, int nBatch, cudaStream_t st, int cpb,
                         long hBatch, int hDiv, const int *hMap) {
  cpb = std::min(cpb > 0 ? cpb : 4, cols2_cpb(f, 8));
  allow_max_smem((const void *)k_cols2);
  const int threads = (cpb * std::max(f.R1, f.R2) + 31) / 32 * 32;
  return launch_pdl(k_cols2, dim3((nColsC + cpb - 1) / cpb, nBatch), dim3(threads), cols2_smem(f, cpb), st,
                    reinterpret_cast<cplx<float> *>(spec), pitch, batch, nColsC, nRowsIn, nRowsOut,
                    reinterpret_cast<const cplx<float> *>(H), hPitch, f, scale, mode == 2 ? -scale : scale, cpb, hBatch,
                    hDiv, hMap);
}

void cols2_prepare_kernels() { allow_max_smem((const void *)k_cols2); }

}  // namespace imfit
