// clblm_scan.cuh -- kernels of the FFT instrument-function scan (scan.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace clblm {

constexpr int kScanRecord = 65536;          // LPTSMX, clblm_FFT.f90:91
constexpr int kScanHalf = kScanRecord / 2;  // complex points per record
constexpr int kScanMaxEdges = 4;

// The scan's spectral-domain set-up (host arithmetic of clblm_FFTSCN_struct
// and Scntrn, clblm_FFT.f90:352-844, :2070-2190).
struct ScanArgs {
  int jfn;            // scanning function 1..10 (0: no scanning apodization)
  double A;           // C(JFN) * HWHM
  double DX;          // 1 / (N * DV), the path-difference step
  const double* X0;   // path difference at the start of every record (complex index k = j * kScanHalf)
  int64_t nhalf;      // N / 2: complex points 0 .. N/2
  int nedge;          // sinc: the interpolated end points of the rectangle
  int64_t edge_k[kScanMaxEdges];
  double edge_v[kScanMaxEdges];
  int deconv;         // 1: divide by the pre-boxing's transform, Z / sin(Z)
  double deconv_a;    // its width parameter (the boxed DV)
  double floor;       // k_scan_low: the apodization's value past the coefficients it forms
};

__global__ void k_scan_load(const double* s, int64_t off, int64_t ltotal, int M, int64_t ktotal, double fill,
                            double* x, int64_t n);
__global__ void k_scan_apod(ScanArgs a, double2* F);
__global__ void k_scan_sfn(int jfn, double A, double dv, int64_t n, double p1, double p2, double p3, double* y);
__global__ void k_scan_mulnum(const double2* H, int64_t nhalf, double2* F);
// the scan through the low coefficients alone: terms of the expansion about a
// block's centre, threads per CTA
constexpr int kScanTerms = 12, kScanTermsWide = 24, kScanLowThreads = 256;
constexpr int kScanLowRatio = 16, kScanWideRatio = 2;  // M >= ratio K: theta < 0.2, < pi / 2
constexpr int kScanPowers = 256;   // half a block's points with tabulated powers
constexpr int kScanLowK = 16;      // coefficients per CTA of k_scan_low
constexpr int kScanFftR = 32, kScanFftMaxC = 4096, kScanFftThreads = 256;  // parts of a transform, points of one
template <int Terms>
__global__ void __launch_bounds__(kScanLowThreads)
    k_scan_moments(const double* __restrict__ s, int64_t off, int64_t ltotal, int boxed, int64_t ktotal, double fill,
                   double2* __restrict__ mom, int64_t nblk, int B, int64_t M, double2* __restrict__ W);
template <bool Back>
__global__ void __launch_bounds__(kScanFftThreads)
    k_scan_fft(const double2* __restrict__ in, double2* __restrict__ out, const double2* __restrict__ W, int64_t M,
               int64_t K, int logC);
template <int Terms>
__global__ void __launch_bounds__(32 * Terms / 2)
    k_scan_low(ScanArgs a, double fill_n, double scale, int64_t K, int64_t M, int R, const double2* __restrict__ X,
               const double2* __restrict__ W, double2* __restrict__ Z);
// the data that k_scan_expand adds the apodization's floor of
struct ScanFloor {
  double floor, fill;
  const double* s;
  int64_t off, n;  // first point of the data in s; points (means) of them
  int boxed;
};
template <int Terms, bool Floor>
__global__ void __launch_bounds__(kScanLowThreads)
    k_scan_expand(const double2* __restrict__ y, int64_t M, int B, int64_t first, int64_t count,
                  double* __restrict__ out, ScanFloor f);
__global__ void k_scan_out(const double* y, int64_t first, int64_t count, double scale, double* out);

}  // namespace clblm
