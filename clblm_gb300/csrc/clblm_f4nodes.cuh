// clblm_f4nodes.cuh -- the nodes of k_f4_far (f4far.cu), host and device.
//
// A far-wing term 1 / (AL2 + x^2) is carried from NP points of a leaf (32
// points) or tile (128) to all of them by the polynomial through the NP (the
// Chebyshev points, rounded to whole points).  Records keep D points away from
// the leaf, 4 D from the tile.
//   mixed path   NP = 10, D = 48: 3.9e-8 of a term, below its FP32 rounding
//   FP64 path    NP = 16, D = 80: 1.8e-16 of a term from the leaf, 3.1e-16 from
//                the tile (D = 64: 3.5e-15 and 6.2e-15).  The weights of the
//                polynomial (they add up to 1, their magnitudes to 3) are rounded
//                once (factor by factor they were off by 3e-16 and 6e-16 of a
//                term) and carry the sums' differences from one node's, a third
//                of the rounding of the sums themselves.  Against the terms added
//                at the point, in record order, the error of a point is 1.3e-16
//                rms for one to five records (1.2e-16), 1.1e-16 for 30 (1.7e-16)
//                and 1.0e-16 for 300 (4.9e-16).
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

// a * b as the sum of two doubles (Veltkamp's split, Dekker's product)
struct FarPair {
  double hi, lo;
};
constexpr FarPair far_product(double a, double b) {
  const double s = 134217729.;  // 2^27 + 1
  const double a1 = s * a - (s * a - a), a2 = a - a1, b1 = s * b - (s * b - b), b2 = b - b1, p = a * b;
  return {p, ((a1 * b1 - p) + a1 * b2 + a2 * b1) + a2 * b2};
}
// weight of node k at point i (Lagrange)
template <bool Plain>
constexpr double far_weight(bool tile, int k, int i) {
  constexpr int NP = Far<Plain>::NP;
  if (Plain) {
    // numerator and denominator exactly (15 factors below 2^7), their quotient
    // and its remainder
    __int128 num = 1, den = 1;
    for (int j = 0; j < NP; ++j)
      if (j != k) {
        num *= i - far_node(Plain, tile, j);
        den *= far_node(Plain, tile, k) - far_node(Plain, tile, j);
      }
    const double nh = (double)num, nl = (double)(num - (__int128)nh);
    const double dh = (double)den, dl = (double)(den - (__int128)dh);
    const double q = nh / dh;
    const FarPair p = far_product(q, dh);
    return q + ((nh - p.hi) - p.lo + nl - q * dl) / dh;
  }
  double v = 1.;
  for (int j = 0; j < NP; ++j)
    if (j != k)
      v *= (double)(i - far_node(Plain, tile, j)) /
           (double)(far_node(Plain, tile, k) - far_node(Plain, tile, j));
  return v;
}
template <bool Plain>
struct FarWeights {
  double leaf[Far<Plain>::NP][kFarLeaf], tile[Far<Plain>::NP][kFarTilePts];
};
template <bool Plain>
constexpr FarWeights<Plain> far_weights() {
  FarWeights<Plain> w{};
  for (int k = 0; k < Far<Plain>::NP; ++k) {
    for (int i = 0; i < kFarLeaf; ++i) w.leaf[k][i] = far_weight<Plain>(false, k, i);
    for (int i = 0; i < kFarTilePts; ++i) w.tile[k][i] = far_weight<Plain>(true, k, i);
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
CLBLM_HD double far_sub(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dsub_rn(a, b);
#else
  return a - b;
#endif
}

// FP64 path: s + w (v - ref) of a node's sum v, ref the sum of node kFarRef,
// which the caller adds to the total
constexpr int kFarRef = 8;
CLBLM_HD double far_carry(double w, double v, double ref, double s) { return far_fma(w, far_sub(v, ref), s); }

}  // namespace clblm
