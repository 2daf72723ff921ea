// clblm_interpmap.cuh -- interpSpectrum's general-ratio branch
// (clblm_Spectrum.f90:528-565) point by point instead of step by step.
//
// The reference steps the phase P by RATIO = DVout/DVin, a carry of INT(P)
// moving into iIn once P >= 1, and restarts both from the exact wavenumber
// every 2400 output points; per point it uses iIn and the table index
// IP = INT(P*201 + 1.00001).  A thread that replays the 2400 steps waits for
// three dependent binary64 operations a step (560 to 880 us per map on GB300,
// whatever the number of points).  Only iIn and IP are used, both truncations,
// so a point k of a block takes them from X = P0 + k RATIO in 64-bit fixed
// point: iIn0 + INT(X) and the fraction's IP.  The stepped P differs from X's
// fraction by the steps' roundings, below 2^-40 over a block; a point whose X
// or whose IP argument lies within map_tol of an integer is not decided that
// way and takes the values of the replayed steps (coincidences of the two
// grids: their rounding picks the side).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define CLBLM_HD __host__ __device__ __forceinline__
#else
#define CLBLM_HD inline
#endif

namespace clblm {

constexpr int kMapBlock = 2400;  // output points between the restarts

CLBLM_HD uint64_t mulhi64(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
// products and sums rounded on their own on either side
CLBLM_HD double map_add(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dadd_rn(a, b);
#else
  return a + b;
#endif
}
CLBLM_HD double map_mul(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}

CLBLM_HD int map_ip(double P) {
  const int IP = (int)map_add(map_mul(P, 201.), 1.00001);
  return IP < 0 ? 0 : (IP > 202 ? 202 : IP);
}

// the block's P0 and RATIO in fixed point (integer part and 2^-64 fraction)
struct MapLin {
  uint64_t p0, r, tol, tol_ip;
  int64_t i0;     // iIn of the block's first point
  int p0i, ri;
  int replay;     // 1: outside the fixed-point form's range, every point is replayed
  int sticky;     // RATIO >= 0.999: INT(iIn + P) may round up, which stays for the rest of the block
};
CLBLM_HD MapLin map_lin(int64_t i0, double P0, double ratio) {
  MapLin m;
  m.i0 = i0;
  m.replay = (P0 > -0.5 && P0 < 1.0 && ratio > 0. && ratio < 1048576.) ? 0 : 1;
  m.sticky = ratio < 0.999 ? 0 : 1;
  m.p0 = m.r = m.tol = m.tol_ip = 0;
  m.p0i = m.ri = 0;
  if (m.replay) return m;
  const int64_t q = (int64_t)(P0 * 4611686018427387904.);  // 2^62
  m.p0i = (int)(q >> 62);
  m.p0 = (uint64_t)q << 2;
  m.ri = (int)ratio;
  m.r = (uint64_t)((ratio - (double)m.ri) * 18446744073709551616.);
  // 2400 roundings of at most 2^-53 (1 + RATIO), and the fixed point's own; at
  // the carry of a sticky block INT(iIn + P) rounds at iIn's size (below 2^31)
  const uint64_t t = ((uint64_t)1 << 28) + ((uint64_t)m.ri << 24);
  m.tol = m.sticky ? t + ((uint64_t)1 << 43) : t;
  m.tol_ip = 202 * t;
  return m;
}

// (iIn, IP) of point k of the block; false: not decided
CLBLM_HD bool map_point(const MapLin& m, uint32_t k, int64_t* iIn, int* IP) {
  const uint64_t lo = (uint64_t)k * m.r;
  const uint64_t fr = lo + m.p0;
  const int64_t I = (int64_t)k * m.ri + (int64_t)mulhi64(k, m.r) + m.p0i + (fr < lo ? 1 : 0);  // INT of X, X = I + fr
  bool ok = true;
  // an integer >= 1 within tol of X: the carry's side is not known
  if (fr < m.tol) ok = I < 1;
  else if (fr > ~m.tol) ok = I + 1 < 1;
  // IP's argument X' * 201 + 1.00001, X' the fraction (or X itself below 0)
  uint64_t a = mulhi64(fr, 201), b = fr * 201;
  const uint64_t c = 184467440737095ull;  // 0.00001 * 2^64
  const uint64_t f = b + c;
  int64_t t = (int64_t)a + 1 + (f < b ? 1 : 0);
  if (I < 0) t -= 201;  // X in [-1, 0): before the first step only
  if (f < m.tol_ip || f > ~m.tol_ip) ok = false;
  *iIn = m.i0 + (I < 0 ? 0 : I);
  *IP = t < 0 ? 0 : (t > 202 ? 202 : (int)t);
  return ok && m.replay == 0;
}

// leading zeros of a nonzero word
CLBLM_HD int clz32(uint32_t x) {
#ifdef __CUDA_ARCH__
  return __clz((int)x);
#else
  return __builtin_clz(x);
#endif
}

// The reference's steps, for RATIO in [2^-8, 2) in integer arithmetic on
// P * 2^61: P + RATIO is at least 2^-9 then, so a binary64 sum is a multiple
// of 2^-61, and rounding it is rounding the low sh bits of the integer half to
// even, sh from the sum's leading bit (the binary64 chain waits 300 ns a step
// on GB300, this one about 30).
struct MapReplay {
  double P, ratio;
  int64_t iIn;
  uint64_t q, rq;
  int fixed;  // 1: q holds P * 2^61
  CLBLM_HD void start(int64_t i0, double P0, double r) {
    iIn = i0;
    P = P0;
    ratio = r;
    fixed = 0;
    q = 0;
    rq = (r >= 0.00390625 && r < 2.0) ? (uint64_t)(r * 2305843009213693952.) : 0;
  }
  CLBLM_HD double phase() const { return fixed ? (double)q * (1. / 2305843009213693952.) : P; }
  CLBLM_HD void step() {
    if (fixed) {
      const uint64_t s = q + rq;
      const int sh = 11 - clz32((uint32_t)(s >> 32));
      const uint32_t one = 1u << sh;
      const uint32_t up = sh > 0 ? (one >> 1) - 1u + (((uint32_t)s >> sh) & 1u) : 0u;
      const uint64_t v = (s + up) & ~(uint64_t)(one - 1u);
      q = v & (((uint64_t)1 << 61) - 1);
      const int64_t n = (int64_t)(v >> 61);  // INT(P)
      if (ratio >= 0.999 && n > 0 && (q >> 40) == 0x1FFFFF)  // INT(iIn + P) may round up
        iIn = (int64_t)map_add((double)iIn, (double)v * (1. / 2305843009213693952.));
      else
        iIn += n;
      return;
    }
    P = map_add(P, ratio);
    if (P >= 1.0) {
      if (ratio < 0.999) {  // P < 2: INT(iIn + P) = iIn + 1, P - 1 is exact
        iIn += 1;
        P = map_add(P, -1.0);
      } else {
        iIn = (int64_t)map_add((double)iIn, P);
        P = map_add(P, -(double)((int64_t)P));
      }
    }
    if (rq && P >= 0.) {
      q = (uint64_t)(P * 2305843009213693952.);
      fixed = (double)q * (1. / 2305843009213693952.) == P ? 1 : 0;
    }
  }
  // IP of the point: INT(P*201. + 1.00001) in integers (the binary64 argument is
  // within 2^-44 of the exact one), in binary64 nearer an integer than that
  CLBLM_HD int ip() const {
    if (fixed) {
      const uint64_t one = (uint64_t)1 << 53, t = (q >> 8) * 201 + one + 90071992547ull;  // 1.00001 * 2^53
      const uint64_t f = t & (one - 1);
      if (f >= 8192 && f <= one - 8192) return (int)(t >> 53);
    }
    return map_ip(phase());
  }
  // n steps.  Below 0.999 INT(iIn + P) is iIn + 1 and the chain has no binary64
  // operation; at 0.5 <= RATIO < 0.999 a sum below 1 is exact on multiples of
  // 2^-53 and one above 1 rounds to a multiple of 2^-52: a chain of a few
  // integer operations.
  CLBLM_HD void steps(int n) {
    int k = 0;
    const bool below = ratio < 0.999, half = ratio >= 0.5;
    while (k < n && !(fixed && (!below || !half || (q & 255) == 0))) {
      step();
      ++k;
    }
    if (k == n) return;
    if (!below) {
      for (; k < n; ++k) {
        const uint64_t s = q + rq;
        const int sh = 11 - clz32((uint32_t)(s >> 32));
        const uint32_t one = 1u << sh, lo = (uint32_t)s;
        const uint32_t up = (one >> 1) - 1u + ((lo >> sh) & 1u);
        const uint64_t v = (s + (sh > 0 ? up : 0u)) & ~(uint64_t)(one - 1u);
        const uint64_t p = v & (((uint64_t)1 << 61) - 1);
        if ((p >> 40) == 0x1FFFFF) {  // INT(iIn + P) may round up
          step();
          continue;
        }
        iIn += (int64_t)(v >> 61);
        q = p;
      }
      return;
    }
    if (!half) {
      int carries = 0;
      for (; k < n; ++k) {
        const uint64_t s = q + rq;
        const int sh = 11 - clz32((uint32_t)(s >> 32));
        const uint32_t one = 1u << sh, lo = (uint32_t)s;
        const uint32_t up = (one >> 1) - 1u + ((lo >> sh) & 1u);
        const uint64_t v = (s + (sh > 0 ? up : 0u)) & ~(uint64_t)(one - 1u);
        carries += (int)(v >> 61);
        q = v & (((uint64_t)1 << 61) - 1);
      }
      iIn += carries;
      return;
    }
    uint64_t p = q >> 8;
    const uint64_t r = rq >> 8;
    int carries = 0;
    for (; k < n; ++k) {
      const uint64_t s = p + r;
      const uint64_t c = s >> 53;  // 1: a carry
      p = (s + (c & (s >> 1))) & ~c & (((uint64_t)1 << 53) - 1);
      carries += (int)c;
    }
    // (a sum of exactly 2 cannot occur: P < 1 and RATIO < 1)
    q = p << 8;
    iIn += carries;
  }
};

// The flagged (undecided) points of a block, first .. last, from the reference's
// steps: emit(k, iIn, IP).  Where INT(iIn + P) may round up at one of them
// (sticky) iIn stays ahead for the rest of the block: seen at the point after
// it, and only then the rest is replayed as well (point by point, 1.7 us each:
// a gradient's two such blocks of 4700 took 600 us when the rest always was).
template <class Emit>
CLBLM_HD void map_replay(const MapLin& m, double P0, double ratio, const unsigned* flags, int first, int last, int n,
                         const Emit& emit) {
  MapReplay r;
  r.start(m.i0, P0, ratio);
  int k = 0;
  for (int w = first >> 5; w <= last >> 5; ++w) {
    unsigned f = flags[w];
    for (int i = 0; f; ++i, f >>= 1) {
      if (!(f & 1u)) continue;
      const int t = 32 * w + i;
      r.steps(t - k);
      k = t;
      emit(k, (int)r.iIn, r.ip());
      if (!m.sticky || t + 1 >= n || (flags[(t + 1) >> 5] >> ((t + 1) & 31) & 1u)) continue;
      r.steps(1);
      k = t + 1;
      int64_t iIn;
      int IP;
      map_point(m, (uint32_t)k, &iIn, &IP);
      if (iIn == r.iIn) continue;
      for (; k < n; ++k) {
        emit(k, (int)r.iIn, r.ip());
        r.step();
      }
      return;
    }
  }
}

#ifdef __CUDACC__
// The map of one block (first output point J1, wavenumber Vo) by one CTA of
// kMapThreads: every thread decides its points, one thread replays the steps
// up to the last point that was not decided.  A map of 100 layers' grids over
// 100,000 points is bound by its 8 bytes a point.
constexpr int kMapThreads = 128;
__device__ __forceinline__ void interp_map_block(double v1, double dvin, double ratio, int64_t J1, double Vo,
                                                 int64_t nout, int2* __restrict__ map) {
  __shared__ MapLin lin;
  __shared__ double p0;
  __shared__ unsigned flags[(kMapBlock + 31) / 32];
  __shared__ int first, last;  // undecided points
  const int n = (int)min(nout - J1 + 1, (int64_t)kMapBlock);
  if (threadIdx.x == 0) {
    // every product and sum rounded on its own (no FMA contraction): a fused
    // v1 + (iIn-1)*dvin moves P by ~1e-10 and flips the carry at coincidences
    const int64_t iIn = (int64_t)__dadd_rn(__ddiv_rn(__dadd_rn(Vo, -v1), dvin), 1.00001);
    const double Vi = __dadd_rn(v1, __dmul_rn((double)(iIn - 1), dvin));
    p0 = __ddiv_rn(__dadd_rn(Vo, -Vi), dvin);
    lin = map_lin(iIn, p0, ratio);
    first = kMapBlock;
    last = -1;
  }
  for (int k = threadIdx.x; k < (kMapBlock + 31) / 32; k += kMapThreads) flags[k] = 0;
  __syncthreads();
  int2* out = map + (J1 - 1);
  for (int k = threadIdx.x; k < n; k += kMapThreads) {
    int64_t iIn;
    int IP;
    if (map_point(lin, (uint32_t)k, &iIn, &IP)) {
      out[k] = make_int2((int)iIn, IP);
    } else {
      atomicOr(&flags[k >> 5], 1u << (k & 31));
      atomicMin(&first, k);
      atomicMax(&last, k);
    }
  }
  __syncthreads();
  if (threadIdx.x != 0 || last < 0) return;
  map_replay(lin, p0, ratio, flags, first, last, n,
             [&](int k, int iIn, int IP) { out[k] = make_int2(iIn, IP); });
}
#endif

}  // namespace clblm
