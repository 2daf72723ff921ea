// Host check of the far wings' nodes (clblm_f4nodes.cuh): the error of the
// polynomial and its weights at the least distance, and sums of one to 300
// records through nodes against the same sums record by record, each to long
// double.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "clblm_f4nodes.cuh"

using namespace clblm;
using L = long double;

namespace {
const FarWeights<false> kMixed = far_weights<false>();
const FarWeights<true> kPlain = far_weights<true>();
int bad = 0;
void hold(const char* what, L got, L bound) {
  printf("%s %.3Le (bound %.3Le)\n", what, got, bound);
  if (!(got <= bound)) bad++;
}
int points(bool tile) { return tile ? kFarTilePts : kFarLeaf; }

// largest relative error of 1/x^2, its pole to either side, carried by the weights
L polynomial(bool plain, bool tile) {
  const int n = points(tile), NP = plain ? Far<true>::NP : Far<false>::NP;
  const L D = (plain ? Far<true>::D : Far<false>::D) * (tile ? 4 : 1);
  L worst = 0;
  for (L at : {-D, -1.37L * D, n - 1 + D, n - 1 + 2.1L * D})
    for (int i = 0; i < n; ++i) {
      auto f = [&](int m) { return 1 / ((m - at) * (m - at)); };
      L s = 0;
      for (int k = 0; k < NP; ++k) {
        const double w = plain ? (tile ? kPlain.tile[k][i] : kPlain.leaf[k][i])
                               : (tile ? kMixed.tile[k][i] : kMixed.leaf[k][i]);
        const L ref = plain ? f(far_node(plain, tile, kFarRef)) : 0;
        s += w * (f(far_node(plain, tile, k)) - ref) + (k == 0 ? ref : 0);
      }
      worst = std::fmax(worst, std::fabs(s / f(i) - 1));
    }
  return worst;
}
}  // namespace

int main() {
  // FP32's rounding is 6e-8 (mixed path), a double's 1.1e-16 (FP64 path: 1.8e-16
  // and 3.1e-16 of the polynomial, and weights to half a unit, magnitudes adding
  // up to 3, of differences up to 0.9 of the term)
  hold("mixed leaf", polynomial(false, false), 4.0e-8L);
  hold("mixed tile", polynomial(false, true), 4.0e-8L);
  hold("fp64 leaf", polynomial(true, false), 4.0e-16L);
  hold("fp64 tile", polynomial(true, true), 5.5e-16L);

  std::mt19937_64 g(5);
  std::uniform_real_distribution<double> u(0., 1.);
  // records within R points of a tile, near records left out
  const int R = 976, T0 = 5000, D = Far<true>::D;
  const double step = 25. / R;
  for (int nrec : {1, 5, 30, 300}) {
    L e_node = 0, e_direct = 0;
    long cnt = 0;
    for (int t = 0; t < 3000 / nrec + 10; ++t) {
      std::vector<double> xn(nrec), sil(nrec), al2(nrec);
      std::vector<int> far(nrec);
      for (int q = 0; q < nrec; ++q) {
        double c;
        do c = T0 - R + (2. * R + 127.) * u(g);
        while (c > T0 - D && c < T0 + 127 + D);
        xn[q] = c * step;
        sil[q] = std::pow(10., -3. * u(g));
        al2[q] = std::pow(10., -6. + 3. * u(g));
        far[q] = c <= T0 - 4 * D || c >= T0 + 127 + 4 * D;
      }
      auto term = [&](int m, int q) {  // SIL / (AL2 + x^2) at point m, by 1 / x rounded
        const double x = std::fma((double)m, step, -xn[q]);
        return 1. / std::fma(x, x, al2[q]);
      };
      auto nodes = [&](bool tile, int base, double* v) {  // a record per lane, then the lanes
        for (int k = 0; k < 16; ++k) {
          double s[32] = {};
          for (int q = 0; q < nrec; ++q)
            if (far[q] == (int)tile) s[q % 32] = std::fma(sil[q], term(base + far_node(true, tile, k), q), s[q % 32]);
          for (int h = 16; h; h /= 2)
            for (int l = 0; l < h; ++l) s[l] += s[l + h];
          v[k] = s[0];
        }
      };
      double vt[16], vl[4][16];
      nodes(true, T0, vt);
      for (int l = 0; l < 4; ++l) nodes(false, T0 + kFarLeaf * l, vl[l]);
      for (int i = 0; i < kFarTilePts; ++i) {
        L e = 0;
        double d = 0.;
        for (int q = 0; q < nrec; ++q) {
          const L x = (L)(T0 + i) * (L)step - (L)xn[q];
          e += (L)sil[q] / (x * x + (L)al2[q]);
          const double xd = std::fma((double)(T0 + i), step, -xn[q]);
          d += sil[q] / std::fma(xd, xd, al2[q]);
        }
        double s = 0.;
        const double* a = vl[i / kFarLeaf];
        for (int k = 0; k < 16; ++k) s = far_carry(kPlain.tile[k][i], vt[k], vt[kFarRef], s);
        for (int k = 0; k < 16; ++k) s = far_carry(kPlain.leaf[k][i % kFarLeaf], a[k], a[kFarRef], s);
        const L rn = (s + (vt[kFarRef] + a[kFarRef])) / e - 1, rd = d / e - 1;
        e_node += rn * rn;
        e_direct += rd * rd;
        cnt++;
      }
    }
    char name[64];
    snprintf(name, sizeof name, "%d records, rms through nodes", nrec);
    // no larger than record by record (for a few records: within a fifth of a rounding, 2^-53 / 5)
    hold(name, std::sqrt(e_node / cnt), std::sqrt(e_direct / cnt) + (nrec <= 5 ? 2.2e-17L : 0.L));
  }
  printf("violations %d\n", bad);
  return bad != 0;
}
