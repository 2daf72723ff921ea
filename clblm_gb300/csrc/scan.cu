// scan.cu -- kernels of the FFT instrument-function scan (clblm_FFTSCN,
// clblm_FFT.f90:352-844) around cuFFT's real transforms:
//
//   k_scan_load  the spectrum from V1Z, padded with FILL to N = LREC*65536
//                points (LoadSpect :1113-1290); with pre-boxing, the means of
//                M consecutive points instead (Boxcar :862-1012, sums in
//                the reference's order)
//   k_scan_apod  the transform times the apodization of the scanning
//                function, computed analytically at the reference's path
//                differences x = X0(record) + k*DX (Scntrn IVX = 1
//                :2170-2185, Scnfnt :1445-1930), then, with pre-boxing,
//                times Z/sin(Z) (function -1, :1935-1958); the Nyquist
//                point is zeroed as the packed first element's imaginary slot
//                of the apodization is
//   k_scan_sfn   IVX = -1: the scanning function sampled at DV in the
//                transform's circular layout (Scntrn :2097-2140, Scnfnt
//                IAPSC = -1), to be transformed by cuFFT
//   k_scan_mulnum  the spectrum's transform times that transform over its
//                first coefficient (the area: Scntrn :2145-2163, Multrn)
//   k_scan_out   the scanned points from N1 on (wrtSpect :2201-2308), with
//                the 1/N of the inverse transform
//
// and, for the apodizations that end (the sinc's rectangle, Beer, Hamming,
// ...; the Gaussian's, below e^-34) well before the transform's last
// path difference, without the transform of all N points: an instrument's
// 0.8 cm are 2000 of the 4 million coefficients of a 3e-4 cm-1 grid.  With N
// points in M blocks of B, block b's point at t in [-1, 1] from its centre,
//   exp(-2 pi i k n / N) = phase(k, b) exp(-i theta t),  theta = pi k / M,
// and exp(-i theta t) = sum_p (-i theta)^p / p! t^p: 12 terms below 1e-16 for
// theta < 0.2 (M >= 16 K), or 24 of them for theta < pi / 2 (M >= 2 K, where
// 16 K leaves blocks of fewer than 32 points), so, of 12,
//   k_scan_moments     sum_j x_j t_j^p of each block, p = 0 .. 11
//   k_scan_fft<false>  their transforms of M points, two moments as one complex
//   k_scan_low         the coefficients k < K from them, times the apodization,
//                      and the 12 spectra of the way back, (i theta)^p / p! of
//                      each (the block centres' phases cancel)
//   k_scan_fft<true>   their transforms
//   k_scan_expand      sum_p t^p Y_p(b) at the scanned points
// The spectrum is read once and the scanned points written once; a 2^23-point
// scan took 2.0 ms, nearly all of it in the transforms' passes over memory.
// The Gaussian does not reach zero: its exponent stops at -34, so that every
// coefficient past K keeps e^-34 = 1.7e-15 of itself.  The transforms carry the
// Gaussian less that floor and k_scan_expand adds the floor times the data (the
// Nyquist coefficient, which the reference drops, with them: below the rounding
// of a transform): 790 -> 798 us for 2,000,000 points, 2070 -> 2140 us for
// 7,000,000.  Deconvolved, where the floor is not a constant, the whole transform
// serves.
#include <cuda_runtime.h>

#include "clblm_scan.cuh"

namespace clblm {

__global__ void k_scan_load(const double* __restrict__ s, int64_t off, int64_t ltotal, int M, int64_t ktotal,
                            double fill, double* __restrict__ x, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double v = fill;
    if (M <= 1) {
      if (i < ltotal) v = s[off + i];
    } else if (i < ktotal) {
      double sum = 0.0;
      for (int m = 0; m < M; ++m) sum = __dadd_rn(sum, s[off + i * M + m]);
      v = __ddiv_rn(sum, (double)M);
    }
    x[i] = v;
  }
}

// apodization of scanning function jfn at path difference x (A = C*HWHM)
__device__ __forceinline__ double apod(int jfn, double x, double A) {
  const double PI = 3.141592653589793;  // 2*ASIN(1.0)
  switch (jfn) {
    case 1: {  // triangle -> sinc**2
      if (x == 0.0) return 1.0;
      const double z = __dmul_rn(__dmul_rn(PI, x), A);
      const double q = __ddiv_rn(sin(z), z);
      return __dmul_rn(q, q);
    }
    case 2: {  // Gaussian
      const double z = __dmul_rn(__dmul_rn(PI, x), A);
      const double e = __dmul_rn(2.0, __dmul_rn(z, z));
      return exp(-(e < 34.0 ? e : 34.0));
    }
    case 3:  // sinc**2 -> triangle
      return x < __ddiv_rn(1.0, A) ? __dadd_rn(1.0, -__dmul_rn(x, A)) : 0.0;
    case 4:  // sinc -> rectangle (end point set separately)
      return x < __ddiv_rn(1.0, A) ? 1.0 : 0.0;
    case 5: {  // Beer
      if (!(x < __ddiv_rn(1.0, A))) return 0.0;
      const double u = __dmul_rn(x, A);
      const double w = __dadd_rn(1.0, -__dmul_rn(u, u));
      return __dmul_rn(w, w);
    }
    case 6:  // Hamming
      if (!(x < __ddiv_rn(1.0, A))) return 0.0;
      return __dmul_rn(0.53835685, __dadd_rn(1.0, __dmul_rn(0.857504, cos(__dmul_rn(__dmul_rn(PI, x), A)))));
    case 7:  // Hanning
      if (!(x < __ddiv_rn(1.0, A))) return 0.0;
      return __dmul_rn(0.5, __dadd_rn(1.0, cos(__dmul_rn(__dmul_rn(PI, x), A))));
    case 8:
    case 9:
    case 10: {  // Norton-Beer weak, medium, strong (:1774-1813)
      if (!(x < __ddiv_rn(1.0, A))) return 0.0;
      const double xa = __dmul_rn(x, A);
      const double u = __dadd_rn(1.0, -__dmul_rn(xa, xa));
      const double u2 = __dmul_rn(u, u);
      if (jfn == 8) return __dadd_rn(__dadd_rn(0.384093, -__dmul_rn(0.087577, u)), __dmul_rn(0.703484, u2));
      if (jfn == 9) return __dadd_rn(__dadd_rn(0.152442, -__dmul_rn(0.136176, u)), __dmul_rn(0.983734, u2));
      return __dadd_rn(__dadd_rn(0.045355, __dmul_rn(0.554883, u2)), __dmul_rn(0.399782, __dmul_rn(u2, u2)));
    }
    default:
      return 1.0;  // boxcar only: no apodization
  }
}

__global__ void k_scan_apod(ScanArgs a, double2* __restrict__ F) {
  const double PI = 3.141592653589793;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k <= a.nhalf;
       k += (int64_t)gridDim.x * blockDim.x) {
    double2 f = F[k];
    if (k == a.nhalf) {  // Nyquist
      F[k] = make_double2(0.0, 0.0);
      continue;
    }
    const int64_t j = k / kScanHalf, kk = k - j * kScanHalf;
    const double x = __dadd_rn(a.X0[j], __dmul_rn((double)kk, a.DX));
    if (a.jfn > 0) {
      double h = apod(a.jfn, x, a.A);
      for (int e = 0; e < a.nedge; ++e)
        if (k == a.edge_k[e]) h = a.edge_v[e];
      f.x = __dmul_rn(f.x, h);
      f.y = __dmul_rn(f.y, h);
    }
    if (a.deconv) {
      const double z = __dmul_rn(__dmul_rn(__dmul_rn(2.0, PI), x), a.deconv_a);
      const double d = z != 0.0 ? __ddiv_rn(z, sin(z)) : 1.0;
      f.x = __dmul_rn(f.x, d);
      f.y = __dmul_rn(f.y, d);
    }
    F[k] = f;
  }
}

// the scanning function of JFN at wavenumber offset x (Scnfnt, IAPSC = -1,
// clblm_FFT.f90:1499-1921)
__device__ double scan_fn(int jfn, double x, double A, double p1, double p2, double p3) {
  const double PI = 3.141592653589793;  // 2*ASIN(1.0)
  const double PI2 = __dmul_rn(2.0, PI);
  switch (jfn) {
    case 1:  // triangle
      return x > A ? 0.0 : __dadd_rn(1.0, -__ddiv_rn(x, A));
    case 2: {  // Gaussian
      const double q = __ddiv_rn(x, A);
      const double e = __dmul_rn(0.5, __dmul_rn(q, q));
      return exp(-(e < 34.0 ? e : 34.0));
    }
    case 3: {  // sinc**2
      if (x == 0.0) return 1.0;
      const double z = __ddiv_rn(__dmul_rn(PI, x), A);
      const double q = __ddiv_rn(sin(z), z);
      return __dmul_rn(q, q);
    }
    case 4: {  // sinc
      if (x == 0.0) return 1.0;
      const double z = __ddiv_rn(__dmul_rn(PI2, x), A);
      return __ddiv_rn(sin(z), z);
    }
    case 5: {  // Beer
      const double u = __ddiv_rn(__dmul_rn(PI2, x), A);
      const double u2 = __dmul_rn(u, u);
      if (u >= 0.5) {
        const double u5 = __dmul_rn(__dmul_rn(u2, u2), u);
        const double t = __dadd_rn(__dmul_rn(__dadd_rn(3.0, -u2), sin(u)), -__dmul_rn(__dmul_rn(3.0, u), cos(u)));
        return __ddiv_rn(__dmul_rn(15., t), u5);
      }
      return __dadd_rn(1.0, -__dmul_rn(15.0 / 210, u2));
    }
    case 6:
    case 7: {  // Hamming, Hanning
      const double c = jfn == 6 ? 0.428752 : 0.5;
      const double u = __ddiv_rn(__dmul_rn(PI2, x), A);
      if (u == 0.0) return 1.0;
      if (fabs(u) == PI) return c;
      const double up = __dadd_rn(u, PI), um = __dadd_rn(u, -PI);
      return __dadd_rn(__ddiv_rn(sin(u), u), __dmul_rn(c, __dadd_rn(__ddiv_rn(sin(up), up), __ddiv_rn(sin(um), um))));
    }
    case 13: {  // Kiruna: sinc at 0 and at the offset p1, weights p2 and p3
      const double u1 = __ddiv_rn(__dmul_rn(PI2, x), A);
      const double u2 = __ddiv_rn(__dmul_rn(PI2, __dadd_rn(x, -p1)), A);
      const double f1 = u1 == 0.0 ? 1.0 : __ddiv_rn(sin(u1), u1);
      const double f2 = u2 == 0.0 ? 1.0 : __ddiv_rn(sin(u2), u2);
      return __dadd_rn(__dmul_rn(p2, f1), __dmul_rn(p3, f2));
    }
    default:
      return 0.0;
  }
}

__global__ void k_scan_sfn(int jfn, double A, double dv, int64_t n, double p1, double p2, double p3,
                           double* __restrict__ y) {
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < n; g += (int64_t)gridDim.x * blockDim.x) {
    double x;
    if (jfn == 13 && g >= n / 2) {  // the negative blocks as the reference writes them
      const int64_t ng = n - g;
      const int64_t J = (ng + kScanRecord - 1) / kScanRecord;
      x = __dmul_rn((double)((2 * J - 2) * kScanRecord - ng + 2), dv);
    } else {
      x = __dmul_rn((double)(g < n - g ? g : n - g), dv);
    }
    y[g] = scan_fn(jfn, x, A, p1, p2, p3);
  }
}

__global__ void k_scan_mulnum(const double2* __restrict__ H, int64_t nhalf, double2* __restrict__ F) {
  const double factor = H[0].x;  // the scanning function's area
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k <= nhalf; k += (int64_t)gridDim.x * blockDim.x) {
    const double2 h = H[k];
    const double hx = __ddiv_rn(h.x, factor), hy = __ddiv_rn(h.y, factor);
    const double2 f = F[k];
    F[k] = make_double2(__dadd_rn(__dmul_rn(f.x, hx), -__dmul_rn(f.y, hy)),
                        __dadd_rn(__dmul_rn(f.x, hy), __dmul_rn(f.y, hx)));
  }
}

// point i of the data: the spectrum's own or, pre-boxed, the mean of `boxed`
__device__ __forceinline__ double scan_point(const double* __restrict__ s, int64_t off, int boxed, int64_t i) {
  if (boxed <= 1) return s[off + i];
  double sum = 0.0;
  for (int m = 0; m < boxed; ++m) sum = __dadd_rn(sum, s[off + i * boxed + m]);
  return __ddiv_rn(sum, (double)boxed);
}

// t_j^(2q) of a block's lower half (q = 0: t itself) in shared memory
__device__ __forceinline__ void scan_powers(int B, double (*T)[kScanPowers], int n) {
  const double rh = 2. / (double)B, c = 0.5 * (double)(B - 1);
  for (int j = threadIdx.x; j < B / 2; j += blockDim.x) {
    const double t = ((double)j - c) * rh, t2 = t * t;
    T[0][j] = t;
    double e = t2;
    for (int q = 1; q < n; ++q) {
      T[q][j] = e;
      e *= t2;
    }
  }
  __syncthreads();
}

// moments of a block of B points (even): the pairs (j, B-1-j), whose t are
// opposite, over the kMomLanes lanes of a block; the FP64 unit bounds it (17
// instructions a pair), so the powers of t come from a table and
// a lane group is as small as the reduction's 16 values allow (lane q ends
// with moments 2q and 2q+1, or four of 24): 77 -> 60 us on 2,000,000 points against a warp
// per block and powers by multiplication.  The blocks past the data are
// zeroed, and W gets exp(-2 pi i j / M) for the transforms.
template <int Terms>
__global__ void __launch_bounds__(kScanLowThreads)
    k_scan_moments(const double* __restrict__ s, int64_t off, int64_t ltotal, int boxed, int64_t ktotal, double fill,
                   double2* __restrict__ mom, int64_t nblk, int B, int64_t M, double2* __restrict__ W) {
  constexpr int kMomLanes = 8, kSums = Terms <= 16 ? 16 : 32, kMine = kSums / kMomLanes;
  __shared__ double T[Terms / 2][kScanPowers];
  const bool table = B / 2 <= kScanPowers;
  if (table) scan_powers(B, T, Terms / 2);
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nthr = (int64_t)gridDim.x * blockDim.x;
  const int lane = threadIdx.x & (kMomLanes - 1);
  const int64_t n = boxed <= 1 ? ltotal : ktotal;
  auto value = [&](int64_t i) -> double {  // less FILL, which reaches k = 0 alone
    if (i >= n) return 0.;
    const double x = scan_point(s, off, boxed, i);
    return fill != 0. ? __dadd_rn(x, -fill) : x;
  };
  const double rh = 2. / (double)B, c = 0.5 * (double)(B - 1);
  // (whole warps: the last one's spare groups take block M - 1 again)
  const int64_t groups = (M * kMomLanes + 31) / 32 * (32 / kMomLanes);
  for (int64_t g = tid / kMomLanes; g < groups; g += nthr / kMomLanes) {
    const int64_t b = g < M ? g : M - 1;
    double v[kSums];
#pragma unroll
    for (int p = 0; p < kSums; ++p) v[p] = 0.;
    if (b < nblk) {
      const int64_t i0 = b * B;
      if (table) {
#pragma unroll 4
        for (int j = lane; j < B / 2; j += kMomLanes) {
          const double x0 = value(i0 + j), x1 = value(i0 + B - 1 - j);
          const double e = x0 + x1, o = (x0 - x1) * T[0][j];  // (t of the other point is -t)
          v[0] += e;
          v[1] += o;
#pragma unroll
          for (int q = 1; q < Terms / 2; ++q) {
            v[2 * q] = fma(e, T[q][j], v[2 * q]);
            v[2 * q + 1] = fma(o, T[q][j], v[2 * q + 1]);
          }
        }
      } else {
        for (int j = lane; j < B / 2; j += kMomLanes) {
          const double x0 = value(i0 + j), x1 = value(i0 + B - 1 - j);
          const double t = ((double)j - c) * rh, t2 = t * t;
          double e = x0 + x1, o = (x0 - x1) * t;
#pragma unroll
          for (int p = 0; p < Terms; p += 2) {
            v[p] += e;
            v[p + 1] += o;
            e *= t2;
            o *= t2;
          }
        }
      }
    }
    // totals over the lanes: lane l ends with those of v[kMine l ..]
#pragma unroll
    for (int h = kSums / 2; h >= kMine; h >>= 1) {
      const bool up = (lane & (h / kMine)) != 0;
#pragma unroll
      for (int i = 0; i < h; ++i) {
        const double send = up ? v[i] : v[i + h];
        const double keep = up ? v[i + h] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, h / kMine);
      }
    }
#pragma unroll
    for (int i = 0; i < kMine / 2; ++i) {
      const int q = lane * (kMine / 2) + i;
      if (q < Terms / 2) mom[(int64_t)q * M + b] = make_double2(v[2 * i], v[2 * i + 1]);
    }
  }
  if (W)
    for (int64_t j = tid; j < M; j += nthr) {
      double sn, cs;
      sincospi(2. * (double)j / (double)M, &sn, &cs);
      W[j] = make_double2(cs, -sn);
    }
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }

// One transform of C = M / kScanFftR points per CTA: the part r (mod kScanFftR)
// of an M-point transform of which only the coefficients |k| < K are wanted.
// Forward:
//   X_r[j] = sum_c z[r + R c] w_C^(j c), so that X[k] = sum_r w_M^(r k) X_r[k mod C]
// (the sum over r in k_scan_low); way back, from the Z[k] of |k| < K alone:
//   y[r + R c] = sum_j conj(w_C)^(j c) sum_{k = j mod C} conj(w_M)^(r k) Z[k].
// Radix-4 Stockham passes (Stockham's autosort transform) in shared memory.
// The 6 transforms of M = 32768 points were 255 us each way as 12 real ones of
// a library with a CTA per transform (12 of 152 SMs); 192 CTAs take 27 us
// forward and 39 back (FP64 unit, and 40 SMs with a second CTA).
// The parts' number is fixed, so that the sum over r stays 32 terms; above
// kScanFftMaxC points a part, M is enough work for the library's transforms.
template <bool Back>
__global__ void __launch_bounds__(kScanFftThreads)
    k_scan_fft(const double2* __restrict__ in, double2* __restrict__ out, const double2* __restrict__ W, int64_t M,
               int64_t K, int logC) {
  extern __shared__ double2 sm[];
  const int C = 1 << logC, r = blockIdx.x;
  double2 *x = sm, *y = sm + C, *w = sm + 2 * C;
  const int64_t row = (int64_t)blockIdx.y * M;
  for (int j = threadIdx.x; j < C; j += blockDim.x) {
    const double2 wc = W[(int64_t)j * kScanFftR];
    w[j] = Back ? cconj(wc) : wc;
    if (!Back) {
      x[j] = in[row + r + (int64_t)kScanFftR * j];
    } else {
      double2 u = make_double2(0., 0.);
      for (int64_t k = j; k < K; k += C) {
        const double2 t = cmul(in[row + k], cconj(W[(r * k) & (M - 1)]));
        u.x += t.x;
        u.y += t.y;
      }
      for (int64_t k = C - j; k < K; k += C) {  // -k = j mod C
        const double2 t = cmul(in[row + M - k], W[(r * k) & (M - 1)]);
        u.x += t.x;
        u.y += t.y;
      }
      x[j] = u;
    }
  }
  __syncthreads();
  int ls = 0;  // log2 of the stride
  for (; logC - ls >= 2; ls += 2) {
    const int s = 1 << ls, quarter = C >> 2;
    for (int t = threadIdx.x; t < quarter; t += blockDim.x) {
      const int q = t & (s - 1), ps = t - q;  // ps = p * s
      const double2 a = x[t], b = x[t + quarter], c = x[t + 2 * quarter], d = x[t + 3 * quarter];
      const double2 apc = make_double2(a.x + c.x, a.y + c.y), amc = make_double2(a.x - c.x, a.y - c.y);
      const double2 bpd = make_double2(b.x + d.x, b.y + d.y), bmd = make_double2(b.x - d.x, b.y - d.y);
      // -i (b - d) forward, i (b - d) back
      const double2 jd = Back ? make_double2(-bmd.y, bmd.x) : make_double2(bmd.y, -bmd.x);
      double2* o = y + q + 4 * ps;
      o[0] = make_double2(apc.x + bpd.x, apc.y + bpd.y);
      o[s] = cmul(w[ps], make_double2(amc.x + jd.x, amc.y + jd.y));
      o[2 * s] = cmul(w[2 * ps], make_double2(apc.x - bpd.x, apc.y - bpd.y));
      o[3 * s] = cmul(w[3 * ps], make_double2(amc.x - jd.x, amc.y - jd.y));
    }
    __syncthreads();
    double2* z = x;
    x = y;
    y = z;
  }
  if (logC - ls == 1) {
    const int s = 1 << ls;
    for (int t = threadIdx.x; t < s; t += blockDim.x) {
      const double2 a = x[t], b = x[t + s];
      y[t] = make_double2(a.x + b.x, a.y + b.y);
      y[t + s] = make_double2(a.x - b.x, a.y - b.y);
    }
    __syncthreads();
    x = y;
  }
  for (int j = threadIdx.x; j < C; j += blockDim.x) {
    if (Back) out[row + r + (int64_t)kScanFftR * j] = x[j];
    else out[row + (int64_t)r * C + j] = x[j];
  }
}

// Coefficients k < K of the spectrum from the transforms of its moments, times
// the apodization (k_scan_apod's) and `scale`, and the spectra of the way
// back: pair q = (moments 2q, 2q+1) by warp q, 16 k's by halves of the parts.
// With z = m_2q + i m_(2q+1), A = Z[k] and D = conj(Z[M-k]), a and b the
// theta^p / p! of the two moments and s = (-1)^q, the pair adds
//   s/2 ((a - b) A + (a + b) D)
// to the coefficient w, and y_2q + i y_(2q+1) has the spectrum s (a - b) w at
// k, s (a + b) conj(w) at -k.  R = kScanFftR parts (k_scan_fft), or 1 part (W
// not read).
template <int Terms>
__global__ void __launch_bounds__(32 * Terms / 2)
    k_scan_low(ScanArgs a, double fill_n, double scale, int64_t K, int64_t M, int R, const double2* __restrict__ X,
               const double2* __restrict__ W, double2* __restrict__ Z) {
  const double PI = 3.141592653589793;
  __shared__ double2 part[Terms / 2][kScanLowK], tot[kScanLowK];
  const int q = threadIdx.x >> 5, lane = threadIdx.x & 31, kl = lane & (kScanLowK - 1);
  const int64_t k = (int64_t)blockIdx.x * kScanLowK + kl;
  const bool in = k < K;
  const int64_t C = M / R, kc = k & (C - 1), kn = (C - kc) & (C - 1);
  double2 A = make_double2(0., 0.), D = make_double2(0., 0.);
  const double2* x = X + (int64_t)q * M;
  if (in) {
    if (R == 1) {
      if (lane < kScanLowK) {
        A = x[kc];
        D = cconj(x[kn]);
      }
    } else {
#pragma unroll 8
      for (int i = 0; i < kScanFftR / 2; ++i) {
        const int r = i + (lane / kScanLowK) * (kScanFftR / 2);
        const double2 w = W[(r * k) & (M - 1)], f = x[r * C + kc], g = x[r * C + kn];
        A.x = fma(w.x, f.x, fma(-w.y, f.y, A.x));
        A.y = fma(w.x, f.y, fma(w.y, f.x, A.y));
        D.x = fma(w.x, g.x, fma(w.y, g.y, D.x));
        D.y = fma(-w.x, g.y, fma(w.y, g.x, D.y));
      }
    }
  }
  A.x += __shfl_xor_sync(0xffffffffu, A.x, kScanLowK);
  A.y += __shfl_xor_sync(0xffffffffu, A.y, kScanLowK);
  D.x += __shfl_xor_sync(0xffffffffu, D.x, kScanLowK);
  D.y += __shfl_xor_sync(0xffffffffu, D.y, kScanLowK);
  const double th = PI * (double)k / (double)M;
  double ca = 1., cb = th;  // theta^p / p! of p = 2q and 2q + 1
  for (int p = 1; p <= q; ++p) {
    ca = ca * (th * th) * (1. / (double)((2 * p - 1) * (2 * p)));
    cb = cb * (th * th) * (1. / (double)((2 * p) * (2 * p + 1)));
  }
  const double sg = q & 1 ? -1. : 1., cm = sg * (ca - cb), cp = sg * (ca + cb);
  if (lane < kScanLowK)
    part[q][kl] = make_double2(0.5 * (cm * A.x + cp * D.x), 0.5 * (cm * A.y + cp * D.y));
  __syncthreads();
  if (q == 0 && lane < kScanLowK && in) {
    double wr = 0., wi = 0.;
#pragma unroll
    for (int p = 0; p < Terms / 2; ++p) {
      wr += part[p][kl].x;
      wi += part[p][kl].y;
    }
    if (k == 0) wr += fill_n;
    const int64_t j = k / kScanHalf, kk = k - j * kScanHalf;
    const double xd = __dadd_rn(a.X0[j], __dmul_rn((double)kk, a.DX));
    double h = apod(a.jfn, xd, a.A) - a.floor;  // (k_scan_expand adds the floor)
    for (int e = 0; e < a.nedge; ++e)
      if (k == a.edge_k[e]) h = a.edge_v[e];
    wr *= h;
    wi *= h;
    if (a.deconv) {
      const double z = __dmul_rn(__dmul_rn(__dmul_rn(2.0, PI), xd), a.deconv_a);
      const double d = z != 0.0 ? __ddiv_rn(z, sin(z)) : 1.0;
      wr *= d;
      wi *= d;
    }
    tot[kl] = make_double2(wr * scale, wi * scale);
  }
  __syncthreads();
  if (lane < kScanLowK && in) {
    const double2 w = tot[kl];
    Z[(int64_t)q * M + k] = make_double2(cm * w.x, cm * w.y);
    if (k > 0) Z[(int64_t)q * M + M - k] = make_double2(cp * w.x, -cp * w.y);
  }
}

// The scanned points [first, first + count): a warp per block, a lane per
// pair of opposite points (13 FP64 instructions a pair bound it; 42 -> 33 us
// with t from a table and the scale in the coefficients).  Floor: the
// apodization's value at every coefficient that the transforms leave out, which
// multiplies the data themselves (FILL past them).
template <int Terms, bool Floor>
__global__ void __launch_bounds__(kScanLowThreads)
    k_scan_expand(const double2* __restrict__ y, int64_t M, int B, int64_t first, int64_t count,
                  double* __restrict__ out, ScanFloor f) {
  __shared__ double T[2][kScanPowers];
  const bool table = B / 2 <= kScanPowers;
  if (table) scan_powers(B, T, 2);
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const int64_t b0 = first / B, b1 = (first + count - 1) / B;
  const double rh = 2. / (double)B, c = 0.5 * (double)(B - 1);
  for (int64_t b = b0 + (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); b <= b1; b += warps) {
    double2 Y[Terms / 2];
#pragma unroll
    for (int q = 0; q < Terms / 2; ++q) Y[q] = y[(int64_t)q * M + b];
    for (int j = lane; j < B / 2; j += 32) {
      const double t = table ? T[0][j] : ((double)j - c) * rh, t2 = table ? T[1][j] : t * t;
      double e = Y[Terms / 2 - 1].x, o = Y[Terms / 2 - 1].y;
#pragma unroll
      for (int q = Terms / 2 - 2; q >= 0; --q) {
        e = fma(e, t2, Y[q].x);
        o = fma(o, t2, Y[q].y);
      }
      o *= t;
      const int64_t i0 = b * B + j - first, i1 = b * B + B - 1 - j - first;
      auto floor = [&](int64_t i) -> double {
        if constexpr (!Floor) return 0.;
        else return f.floor * (i + first < f.n ? scan_point(f.s, f.off, f.boxed, i + first) : f.fill);
      };
      if (i0 >= 0 && i0 < count) out[i0] = Floor ? e + o + floor(i0) : e + o;
      if (i1 >= 0 && i1 < count) out[i1] = Floor ? e - o + floor(i1) : e - o;
    }
  }
}

#define CLBLM_MOMENTS_ARGS                                                                              \
  const double* __restrict__, int64_t, int64_t, int, int64_t, double, double2* __restrict__, int64_t, int, \
      int64_t, double2* __restrict__
#define CLBLM_LOW_ARGS                                                                                    \
  ScanArgs, double, double, int64_t, int64_t, int, const double2* __restrict__, const double2* __restrict__, \
      double2* __restrict__
#define CLBLM_EXPAND_ARGS const double2* __restrict__, int64_t, int, int64_t, int64_t, double* __restrict__, ScanFloor
#define CLBLM_SCANFFT_ARGS \
  const double2* __restrict__, double2* __restrict__, const double2* __restrict__, int64_t, int64_t, int
template __global__ void k_scan_moments<kScanTerms>(CLBLM_MOMENTS_ARGS);
template __global__ void k_scan_moments<kScanTermsWide>(CLBLM_MOMENTS_ARGS);
template __global__ void k_scan_low<kScanTerms>(CLBLM_LOW_ARGS);
template __global__ void k_scan_low<kScanTermsWide>(CLBLM_LOW_ARGS);
template __global__ void k_scan_expand<kScanTerms, false>(CLBLM_EXPAND_ARGS);
template __global__ void k_scan_expand<kScanTerms, true>(CLBLM_EXPAND_ARGS);
template __global__ void k_scan_expand<kScanTermsWide, false>(CLBLM_EXPAND_ARGS);
template __global__ void k_scan_expand<kScanTermsWide, true>(CLBLM_EXPAND_ARGS);
template __global__ void k_scan_fft<false>(CLBLM_SCANFFT_ARGS);
template __global__ void k_scan_fft<true>(CLBLM_SCANFFT_ARGS);
#undef CLBLM_MOMENTS_ARGS
#undef CLBLM_LOW_ARGS
#undef CLBLM_EXPAND_ARGS
#undef CLBLM_SCANFFT_ARGS

__global__ void k_scan_out(const double* __restrict__ y, int64_t first, int64_t count, double scale,
                           double* __restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = __dmul_rn(y[first + i], scale);
}

}  // namespace clblm
