// clblm_f4nodes.cuh -- the nodes of k_f4_far (f4far.cu), host and device.
//
// A far-wing term 1 / (AL2 + x^2) is carried from NP points of a leaf (32
// points) or tile (128) to all of them by the polynomial through the NP (the
// Chebyshev points, rounded to whole points).  Records keep D points away from
// the leaf, 4 D from the tile.
//   mixed path   NP = 10, D = 48: 3.9e-8 of a term, below its FP32 rounding
//   FP64 path    NP = 16, D = 80: 1.8e-16 of a term from the leaf, 3.1e-16 from
//                the tile (D = 64: 3.5e-15 and 6.2e-15).  The weights of the
//                polynomial (they add up to 1, their magnitudes to 3) stand as
//                pairs of doubles and the sums over the nodes are compensated:
//                in plain doubles those alone were 1.2e-15 of a term.  Against
//                sums of the terms themselves, in record order, the error of a
//                point is as large for one to five records (1.2e-16 rms) and a
//                fifth of it for 300; the FP64 operations it takes are a
//                thirtieth of the kernel's.
#pragma once

#ifdef __CUDACC__
#define CLBLM_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#define CLBLM_HD inline
#endif

namespace clblm {

constexpr int kFarLeaf = 32, kFarTilePts = 128;

template <bool Plain>
struct Far;
template <>
struct Far<false> {
  static constexpr int NP = 10, D = 48;
};
template <>
struct Far<true> {
  static constexpr int NP = 16, D = 80;
};

#ifdef __CUDACC__
__host__ __device__
#endif
constexpr int far_node(bool plain, bool tile, int k) {
  constexpr int l10[10] = {0, 2, 5, 8, 13, 18, 23, 26, 29, 31};
  constexpr int t10[10] = {1, 7, 19, 35, 54, 73, 92, 108, 120, 126};
  constexpr int l16[16] = {0, 1, 2, 4, 6, 8, 11, 14, 17, 20, 23, 25, 27, 29, 30, 31};
  constexpr int t16[16] = {0, 3, 7, 14, 23, 34, 45, 57, 70, 82, 93, 104, 113, 120, 124, 127};
  return plain ? (tile ? t16[k] : l16[k]) : (tile ? t10[k] : l10[k]);
}

// weights of the NP nodes at each point (Lagrange), mixed path
struct FarWeights {
  double leaf[Far<false>::NP][kFarLeaf], tile[Far<false>::NP][kFarTilePts];
};
constexpr FarWeights far_weights() {
  constexpr int NP = Far<false>::NP;
  FarWeights w{};
  for (int k = 0; k < NP; ++k) {
    for (int i = 0; i < kFarLeaf; ++i) {
      double v = 1.;
      for (int j = 0; j < NP; ++j)
        if (j != k)
          v *= (double)(i - far_node(false, false, j)) /
               (double)(far_node(false, false, k) - far_node(false, false, j));
      w.leaf[k][i] = v;
    }
    for (int i = 0; i < kFarTilePts; ++i) {
      double v = 1.;
      for (int j = 0; j < NP; ++j)
        if (j != k)
          v *= (double)(i - far_node(false, true, j)) / (double)(far_node(false, true, k) - far_node(false, true, j));
      w.tile[k][i] = v;
    }
  }
  return w;
}

// the same, FP64 path, each the sum of two doubles
struct FarPair {
  double hi, lo;
};
struct FarPairs {
  FarPair leaf[Far<true>::NP][kFarLeaf], tile[Far<true>::NP][kFarTilePts];
};
// a * b as the sum of two doubles (Veltkamp's split, Dekker's product)
constexpr FarPair far_product(double a, double b) {
  const double s = 134217729.;  // 2^27 + 1
  const double a1 = s * a - (s * a - a), a2 = a - a1, b1 = s * b - (s * b - b), b2 = b - b1, p = a * b;
  return {p, ((a1 * b1 - p) + a1 * b2 + a2 * b1) + a2 * b2};
}
constexpr FarPair far_pair(bool tile, int k, int i) {
  // numerator and denominator exactly: products of 15 factors below 2^7
  __int128 num = 1, den = 1;
  for (int j = 0; j < Far<true>::NP; ++j)
    if (j != k) {
      num *= i - far_node(true, tile, j);
      den *= far_node(true, tile, k) - far_node(true, tile, j);
    }
  const double nh = (double)num, nl = (double)(num - (__int128)nh);
  const double dh = (double)den, dl = (double)(den - (__int128)dh);
  const double q = nh / dh;
  const FarPair p = far_product(q, dh);
  return {q, ((nh - p.hi) - p.lo + nl - q * dl) / dh};
}
constexpr FarPairs far_pairs() {
  FarPairs w{};
  for (int k = 0; k < Far<true>::NP; ++k) {
    for (int i = 0; i < kFarLeaf; ++i) w.leaf[k][i] = far_pair(false, k, i);
    for (int i = 0; i < kFarTilePts; ++i) w.tile[k][i] = far_pair(true, k, i);
  }
  return w;
}

CLBLM_HD double far_fma(double a, double b, double c) {
#ifdef __CUDA_ARCH__
  return __fma_rn(a, b, c);
#else
  return std::fma(a, b, c);
#endif
}
CLBLM_HD double far_mul(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}
CLBLM_HD double far_add(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dadd_rn(a, b);
#else
  return a + b;
#endif
}

// sum of w_k v_k, the roundings of its products and additions kept beside it
// (Knuth's two-sum; the dot product of Ogita, Rump and Oishi, SIAM J. Sci.
// Comput. 26, 2005)
struct FarSum {
  double s = 0., c = 0.;
  CLBLM_HD void add(double x) {
    const double t = far_add(s, x), b = far_add(t, -s);
    c = far_add(c, far_add(far_add(s, -far_add(t, -b)), far_add(x, -b)));
    s = t;
  }
  CLBLM_HD void add(FarPair w, double v) {
    const double p = far_mul(w.hi, v);
    c = far_fma(w.lo, v, far_add(c, far_fma(w.hi, v, -p)));
    add(p);
  }
  CLBLM_HD double value() const { return far_add(s, c); }
};

}  // namespace clblm
