// Host check of clblm_interpmap.cuh: the points of a block in fixed point with
// the undecided ones replayed, against the reference's steps in binary64.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <random>

#include "clblm_interpmap.cuh"

using namespace clblm;

static long long bad = 0, points = 0, undecided = 0;

static void block(int64_t i0, double P0, double r) {
  const MapLin m = map_lin(i0, P0, r);
  MapReplay rep, far;  // step by step, and in strides as a block's undecided points take them
  rep.start(i0, P0, r);
  far.start(i0, P0, r);
  int at = 0, stride = 1;
  int64_t iIn = i0;
  double P = P0;
  bool from = false;
  // the block's map as the device forms it: decided points, then the others
  static unsigned flags[(kMapBlock + 31) / 32];
  static int64_t wi[kMapBlock];
  static int wp[kMapBlock];
  int first = kMapBlock, last = -1;
  for (unsigned& f : flags) f = 0;
  for (int k = 0; k < kMapBlock; ++k) {
    if (map_point(m, (uint32_t)k, &wi[k], &wp[k])) continue;
    flags[k >> 5] |= 1u << (k & 31);
    first = k < first ? k : first;
    last = k;
  }
  if (last >= 0)
    map_replay(m, P0, r, flags, first, last, kMapBlock, [](int k, int i, int ip) {
      wi[k] = i;
      wp[k] = ip;
    });
  for (int k = 0; k < kMapBlock; ++k) {
    // the reference's step
    const int IPr = (int)(P * 201. + 1.00001);
    const int IP = IPr < 0 ? 0 : (IPr > 202 ? 202 : IPr);
    int64_t gi;
    int gp;
    const bool ok = map_point(m, (uint32_t)k, &gi, &gp);
    if (!ok && m.sticky) from = true;
    if (!ok || from) {
      gi = rep.iIn;
      gp = map_ip(rep.phase());
      undecided++;
    }
    if (k == at + stride || k == kMapBlock - 1) {
      far.steps(k - at);
      at = k;
      stride = stride % 97 + 1;
      if (far.iIn != rep.iIn || far.phase() != rep.phase()) {
        if (bad++ < 5) printf("strides: i0 %lld P0 %.17g r %.17g k %d\n", (long long)i0, P0, r, k);
      }
    }
    points++;
    if ((int)wi[k] != (int)iIn || wp[k] != IP) {
      if (bad++ < 5) printf("block: i0 %lld P0 %.17g r %.17g k %d\n", (long long)i0, P0, r, k);
    }
    if (gi != iIn || gp != IP) {
      if (bad++ < 5) printf("i0 %lld P0 %.17g r %.17g k %d: %lld %d, want %lld %d\n", (long long)i0, P0, r, k, (long long)gi, gp, (long long)iIn, IP);
    }
    P = P + r;
    if (P >= 1.0) {
      iIn = (int64_t)((double)iIn + P);
      P = P - (double)((int64_t)P);
    }
    rep.step();
  }
}

// the blocks of a grid pair, as interpSpectrum restarts them
static void grid(double v1, double dvin, double dvout, int blocks, int first) {
  for (int b = first; b < first + blocks; ++b) {
    const double Vo = b == 0 ? v1 : v1 + (double)((int64_t)b * kMapBlock) * dvout;
    const int64_t iIn = (int64_t)((Vo - v1) / dvin + 1.00001);
    const double Vi = v1 + (double)(iIn - 1) * dvin;
    block(iIn, (Vo - Vi) / dvin, dvout / dvin);
  }
}

int main() {
  std::mt19937_64 g(7);
  std::uniform_real_distribution<double> u(0., 1.);
  for (int k = 0; k < 2000; ++k) {  // any ratio
    const double dvin = std::pow(10., -4. + 3. * u(g)), r = std::pow(2., -8. + 11. * u(g));
    grid(10. + 3000. * u(g), dvin, dvin * r, 2, (int)(500 * u(g)));
  }
  for (int k = 0; k < 4000; ++k) {  // grids with coincidences: DV of a few digits
    const int a = 1 + (int)(2000 * u(g)), b = 1 + (int)(2000 * u(g));
    const double s = std::pow(10., -(double)(4 + (int)(4 * u(g))));
    grid(std::floor(3000. * u(g)) + (k & 1 ? 0. : 0.25), a * s, b * s, 2, (int)(300 * u(g)));
  }
  for (int a = 1; a <= 40; ++a)  // small fractions
    for (int b = 1; b <= 40; ++b) grid(600., 0.001 * a, 0.001 * b, 1, (a * b) % 7);
  for (double r : {0.5, 0.00390625, 0.0039, 1.9999999, 1.5, 1.25, 0.49999, 0.998999, 0.999, 0.9990001, 1. - 1e-9, 1. + 1e-9, 0.25, 0.75, 1.0, 2.0, 3.5, 1e-6, 500.25, 3e6})
    for (double P0 : {0., -1e-5, -1e-12, 1e-12, 0.5, 1. - 1e-5, 1. - 1e-9, -0.6, 1.0})
      for (int64_t i0 : {(int64_t)1, (int64_t)4999999, (int64_t)2000000000}) block(i0, P0, r);
  printf("points %lld undecided %lld mismatches %lld\n", points, undecided, bad);
  return bad != 0;
}
