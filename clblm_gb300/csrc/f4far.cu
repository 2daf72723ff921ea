// f4far.cu -- far-wing function 4 on the DVR4 grid (CNVF4Q,
// clblm_ODLAY_LineF4.f90:187-494) with the distant records evaluated at a few
// points per tile and interpolated.
//
// Every record reaches the points within 25 cm-1 of its line: R = 25 / DVR4
// to either side, 976 at a 0.1 hPa layer, so a column's upper layers sum some
// 6000 records at each point.  Away from the line a record's term
// SIL / (AL2 + x^2) plus its pedestal (a parabola) is smooth on the scale of
// its distance: on a leaf of 32 points, and on a tile of 128 from four times
// the distance, it is a polynomial through NP of them to the path's rounding
// (clblm_f4nodes.cuh).  A CTA of four warps takes a tile, a warp a leaf:
//   - records that keep DB away from the tile and reach all of it: at the
//     tile's NP nodes, a record per lane, shared out among the warps;
//   - the others that keep D away from the leaf and reach all of it: at the
//     leaf's NP nodes, a record per lane;
//   - the rest (near the leaf, or ending inside it): at its 32 points, one per
//     lane, the records passing through shared memory.
// With R = 976 that is 422 evaluations (FP64 path: 690) per unit of record
// density and point instead of 1928.  Node sums are carried to the points
// in binary64.  The index ranges come from the running bounds of the records' centres (their
// order is nearly that of their centres): searches, one per lane.
//
// FP64: reference's terms, one division each (a reciprocal; the reference's
// ZVSQ = x^2/ALV2 <= 64^2 is compared as x^2 <= 64^2 ALV2).  Mixed: packed
// FP32x2 (two records, or two nodes), groups of at most 32 records in FP32,
// compensated between groups, the node sums' lanes added in binary64.
#include <cuda_runtime.h>

#include <type_traits>

#include "clblm_common.cuh"
#include "clblm_f4nodes.cuh"
#include "clblm_fpconv.cuh"
#include "clblm_kernels.cuh"
#include "clblm_panel.cuh"

namespace clblm {

namespace {

constexpr int kLeaf = kFarLeaf, kTileLeaves = kFarTile / kLeaf;
static_assert(kFarTile == kFarTilePts && 32 * kTileLeaves == kFarThreads, "a warp per leaf");

__device__ const FarWeights<false> c_farw_mixed = far_weights<false>();
__device__ const FarWeights<true> c_farw_plain = far_weights<true>();

__device__ __forceinline__ float rcp_f(float x) {  // PTX rcp.approx: relative error < 2^-23
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

struct SumK {  // compensated FP32 sum
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float x) {
    const float y = __fsub_rn(x, c);
    const float t = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(t, s), y);
    s = t;
  }
  __device__ __forceinline__ double value() const { return (double)s - (double)c; }
};

// v[0 .. 15] of every lane summed over the lanes: lane l ends with the total
// of v[l >> 1] (in v[0])
__device__ __forceinline__ double lane_totals(double v[16], int lane) {
#pragma unroll
  for (int h = 8; h >= 1; h >>= 1) {
    const int bit = 2 * h;  // 16, 8, 4, 2
    const bool up = (lane & bit) != 0;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const double send = up ? v[i] : v[i + h];
      const double keep = up ? v[i + h] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// Accumulates the records [i0, i1), a record per lane from i0 + first in
// steps of `step`, at the nodes m0 + node k (mixed path).
struct FarSumF {
  SumK s[10];
  float2 t[5];
  int pend;
  __device__ __forceinline__ FarSumF() : pend(0) {
#pragma unroll
    for (int k = 0; k < 5; ++k) t[k] = make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ void flush() {
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      s[2 * k].add(t[k].x);
      s[2 * k + 1].add(t[k].y);
      t[k] = make_float2(0.f, 0.f);
    }
    pend = 0;
  }
  template <bool Tile>
  __device__ __forceinline__ void add(const F4Rec* __restrict__ recs, int64_t i0, int64_t i1, int first, int step,
                                      int m0, float2 dvr4) {
    for (int64_t i = i0 + first; i < i1; i += step) {
      const float4* q = reinterpret_cast<const float4*>(recs + i);
      const float4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);  // {nmc, x0}, {nfb0, fb2}, {al2, sil}, each twice
      const float dm = (float)m0 + a.x;  // exact: grid indices are below 2^24
      const float2 x0 = make_float2(a.z, a.w), nfb0 = make_float2(b.x, b.y), fb2 = make_float2(b.z, b.w),
                   al2 = make_float2(c.x, c.y), sil = make_float2(c.z, c.w), dm2 = make_float2(dm, dm);
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const float2 off = make_float2((float)far_node(false, Tile, 2 * k), (float)far_node(false, Tile, 2 * k + 1));
        const float2 x = __ffma2_rn(__fadd2_rn(dm2, off), dvr4, x0);
        const float2 xx = __fmul2_rn(x, x);
        const float2 den = __fadd2_rn(xx, al2);
        const float2 f = __ffma2_rn(sil, make_float2(rcp_f(den.x), rcp_f(den.y)), __ffma2_rn(xx, fb2, nfb0));
        t[k] = __fadd2_rn(t[k], f);
      }
      if (++pend == 8) flush();
    }
  }
  template <bool Tile>
  __device__ __forceinline__ double total(int lane, double) {
    flush();
    double v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = k < 10 ? s[k < 10 ? k : 0].value() : 0.;
    return lane_totals(v, lane);
  }
};

// the same on the FP64 path.  The pedestals, parabolas in the node's offset
// from m0, are summed by their coefficients: a node's term is then six
// operations of the FP64 unit, which bounds the kernel, instead of ten.
struct FarSumD {
  double s[16], p0, p1, p2;
  __device__ __forceinline__ FarSumD() : p0(0.), p1(0.), p2(0.) {
#pragma unroll
    for (int k = 0; k < 16; ++k) s[k] = 0.;
  }
  template <bool Tile>
  __device__ __forceinline__ void add(const F4RecD* __restrict__ recs, int64_t i0, int64_t i1, int first, int step,
                                      int m0, double dvr4, double rbnd2) {
    for (int64_t i = i0 + first; i < i1; i += step) {
      const F4RecD d = recs[i];
      const double nfb0 = d.co2 ? -2. * d.fbnd : -d.fbnd, fb2 = d.co2 ? d.fbnd * rbnd2 : 0.;
      const double x0 = fma((double)m0, dvr4, -d.xnui), t = fb2 * x0;
      p0 += fma(t, x0, nfb0);
      p1 += t;
      p2 += fb2;
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        const double x = fma((double)(m0 + far_node(true, Tile, k)), dvr4, -d.xnui);
        s[k] = fma(d.sil, rcp_d(fma(x, x, d.al2)), s[k]);
      }
    }
  }
  template <bool Tile>
  __device__ __forceinline__ double total(int lane, double dvr4) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const double h = (double)far_node(true, Tile, k) * dvr4;
      s[k] += fma(h, fma(h, p2, 2. * p1), p0);
    }
    return lane_totals(s, lane);
  }
};

// a warp's 32 records in shared memory, mixed path: pairs of records, each
// field of the pair side by side (the operands of the packed arithmetic)
struct LeafBufF {
  float4 q0[16];  // nmc, x0
  float4 q1[16];  // nfb0, fb2
  float4 q2[16];  // al2, sil
  float4 q3[16];  // ralv2, sa3
  float2 q4[16];  // sb3
  int4 jj[16];    // jmin of both, jmax of both
};
struct LeafBufD {
  double xnui[32], sil[32], al2[32], nfb0[32], fb2[32], core2[32], sa3[32], sb3[32];
  int2 jj[32];
};

// The records [i0, i1) at the warp's 32 points, one per lane (J: the lane's
// 1-based point).  Core: a line may lie within 64 ALFV of a point (the
// polynomial core), else the Lorentzian wing is certain; Mask: a record may
// end inside the leaf.
template <bool Core, bool Mask>
__device__ __forceinline__ void leaf_direct(LeafBufF& B, const F4Rec* __restrict__ recs, int64_t i0, int64_t i1, int J,
                                            float2 dvr4, SumK& acc) {
  const int lane = threadIdx.x & 31;
  float* q0 = reinterpret_cast<float*>(B.q0);
  float* q1 = reinterpret_cast<float*>(B.q1);
  float* q2 = reinterpret_cast<float*>(B.q2);
  float* q3 = reinterpret_cast<float*>(B.q3);
  float* q4 = reinterpret_cast<float*>(B.q4);
  int* jj = reinterpret_cast<int*>(B.jj);
  const int p = lane >> 1, o = lane & 1;
  const float Jm = (float)(J - 1);  // exact: J < 2^24
  const float2 Jm2 = make_float2(Jm, Jm);
  for (int64_t i = i0; i < i1; i += 32) {
    const int cnt = (int)(i1 - i < 32 ? i1 - i : 32);
    const F4Rec* r = recs + (i + (lane < cnt ? lane : 0));
    const bool in = lane < cnt;
    const float nmc = r->nmc.x, x0 = r->x0.x, nfb0 = in ? r->nfb0.x : 0.f, fb2 = in ? r->fb2.x : 0.f, al2 = r->al2.x,
                sil = in ? r->sil.x : 0.f;
    float ralv2 = 0.f, sa3 = 0.f, sb3 = 0.f;
    int jmin = 0, jmax = 0;
    if (Core) {
      ralv2 = r->ralv2.x;
      sa3 = in ? r->sa3.x : 0.f;
      sb3 = in ? r->sb3.x : 0.f;
    }
    if (Mask) {
      jmin = in ? r->jmin : 1;
      jmax = in ? r->jmax : 0;
    }
    __syncwarp();  // the previous batch has been read
    q0[4 * p + o] = nmc;
    q0[4 * p + 2 + o] = x0;
    q1[4 * p + o] = nfb0;
    q1[4 * p + 2 + o] = fb2;
    q2[4 * p + o] = al2;
    q2[4 * p + 2 + o] = sil;
    if (Core) {
      q3[4 * p + o] = ralv2;
      q3[4 * p + 2 + o] = sa3;
      q4[2 * p + o] = sb3;
    }
    if (Mask) {
      jj[4 * p + o] = jmin;
      jj[4 * p + 2 + o] = jmax;
    }
    __syncwarp();
    float2 t0 = make_float2(0.f, 0.f), t1 = t0;
    const int np = (cnt + 1) >> 1;
#pragma unroll 4
    for (int k = 0; k < np; ++k) {
      const float4 a = B.q0[k], b = B.q1[k], c = B.q2[k];
      const float2 x = __ffma2_rn(__fadd2_rn(Jm2, make_float2(a.x, a.y)), dvr4, make_float2(a.z, a.w));
      const float2 xx = __fmul2_rn(x, x);
      const float2 nfb = __ffma2_rn(xx, make_float2(b.z, b.w), make_float2(b.x, b.y));
      const float2 den = __fadd2_rn(xx, make_float2(c.x, c.y));
      float2 f = __ffma2_rn(make_float2(c.z, c.w), make_float2(rcp_f(den.x), rcp_f(den.y)), nfb);
      if (Core) {
        const float4 e = B.q3[k];
        const float2 zv = __fmul2_rn(xx, make_float2(e.x, e.y));
        const float2 cr = __fadd2_rn(__ffma2_rn(zv, B.q4[k], make_float2(e.z, e.w)), nfb);
        f.x = zv.x <= 4096.f ? cr.x : f.x;
        f.y = zv.y <= 4096.f ? cr.y : f.y;
      }
      if (Mask) {
        const int4 j = B.jj[k];
        f.x = (J >= j.x && J <= j.z) ? f.x : 0.f;
        f.y = (J >= j.y && J <= j.w) ? f.y : 0.f;
      } else if (k == np - 1 && (cnt & 1)) {
        f.y = 0.f;
      }
      if (k & 1) t1 = __fadd2_rn(t1, f);
      else t0 = __fadd2_rn(t0, f);
    }
    const float2 t = __fadd2_rn(t0, t1);
    acc.add(t.x + t.y);
  }
}

template <bool Core, bool Mask>
__device__ __forceinline__ void leaf_direct(LeafBufD& B, const F4RecD* __restrict__ recs, int64_t i0, int64_t i1, int J,
                                            double dvr4, double rbnd2, double& acc) {
  const int lane = threadIdx.x & 31;
  const double ZSQBND = 64. * 64.;
  const double A3 = (1. + 2. * ZSQBND) / ((1. + ZSQBND) * (1. + ZSQBND));
  const double B3 = -1. / ((1. + ZSQBND) * (1. + ZSQBND));
  const double Jm = (double)(J - 1);
  for (int64_t i = i0; i < i1; i += 32) {
    const int cnt = (int)(i1 - i < 32 ? i1 - i : 32);
    F4RecD d;
    if (lane < cnt) d = recs[i + lane];
    __syncwarp();  // the previous batch has been read
    if (lane < cnt) {
      B.xnui[lane] = d.xnui;
      B.sil[lane] = d.sil;
      B.al2[lane] = d.al2;
      B.nfb0[lane] = d.co2 ? -2. * d.fbnd : -d.fbnd;
      B.fb2[lane] = d.co2 ? d.fbnd * rbnd2 : 0.;
      if (Core) {
        B.core2[lane] = ZSQBND * d.alv2;
        B.sa3[lane] = d.siv * A3;
        B.sb3[lane] = (d.siv * B3) / d.alv2;
      }
      if (Mask) B.jj[lane] = make_int2(d.jmin, d.jmax);
    }
    __syncwarp();
#pragma unroll 2
    for (int k = 0; k < cnt; ++k) {
      const double x = fma(Jm, dvr4, -B.xnui[k]);
      const double xx = x * x;
      double f = B.sil[k] * rcp_d(B.al2[k] + xx);
      if (Core && xx <= B.core2[k]) f = fma(xx, B.sb3[k], B.sa3[k]);
      f += fma(xx, B.fb2[k], B.nfb0[k]);
      if (Mask) {
        const int2 j = B.jj[k];
        if (J < j.x || J > j.y) f = 0.;
      }
      acc += f;
    }
  }
}

}  // namespace

template <bool Plain>
__global__ void __launch_bounds__(kFarThreads, Plain ? 4 : 6) k_f4_far(const __grid_constant__ F4Args a) {
  using Real = typename std::conditional<Plain, double, float>::type;
  using Rec = typename std::conditional<Plain, F4RecD, F4Rec>::type;
  using Buf = typename std::conditional<Plain, LeafBufD, LeafBufF>::type;
  constexpr int NP = Far<Plain>::NP;
  __shared__ Buf buf[kTileLeaves];
  __shared__ double nodeB[kTileLeaves][16], nodeA[kTileLeaves][16];

  const int layer = blockIdx.y;
  const LayerPlan& P = a.plans[layer + a.layer0];
  const int T0 = blockIdx.x * kFarTile;
  if (T0 >= P.nptr4 + 2) return;  // whole CTA, before its barrier
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int s0 = T0 + kLeaf * warp, s1 = s0 + kLeaf - 1;  // the leaf's points
  const int m = s0 + lane, J = m + 1;
  const int64_t n = a.nrec[layer + a.layer0], nm = a.nmirror[layer + a.layer0];
  const Rec* recs = reinterpret_cast<const Rec*>(Plain ? (const void*)a.recd : (const void*)a.rec) +
                    (int64_t)layer * a.stride;
  // a record of centre mc (nearest point) reaches every point within Rlo of
  // it, none past Rhi; the core of no line reaches past `core` points
  const double R = P.bound4 / P.dvr4;
  const int Rlo = (int)R - 2, Rhi = (int)R + 3;
  const int core = a.core[layer + a.layer0];
  const int D = max(Far<Plain>::D, core), DB = max(4 * Far<Plain>::D, core);
  int64_t pos = 0;
  if (lane < 10) {
    // leaf: lo, hi, first that reaches all, first near, first far again, first
    // that ends inside; tile: the four of its far ranges
    const int t1 = T0 + kFarTile - 1;
    const int x = lane == 0   ? s0 - Rhi
                  : lane == 1 ? s1 + Rhi + 1
                  : lane == 2 ? s1 - Rlo
                  : lane == 3 ? s0 - D + 1
                  : lane == 4 ? s1 + D
                  : lane == 5 ? s0 + Rlo + 1
                  : lane == 6 ? t1 - Rlo
                  : lane == 7 ? T0 - DB + 1
                  : lane == 8 ? t1 + DB
                              : T0 + Rlo + 1;
    // running max of the centres (0, 3, 5, 7, 9) or running min from the right
    const bool mx = lane == 0 || lane == 3 || lane == 5 || lane == 7 || lane == 9;
    const int* b = (mx ? a.pmax_jmax : a.smin_jmin) + (int64_t)layer * a.stride;
    int64_t h = n;
    while (pos < h) {  // first record with b >= x
      const int64_t mid = (pos + h) >> 1;
      if (b[mid] < x) pos = mid + 1;
      else h = mid;
    }
  }
  auto at = [&](int k) { return __shfl_sync(0xffffffffu, pos, k); };
  const int64_t lo = at(0), hi = max(at(1), lo), e1 = at(2), n1 = at(3), n2 = at(4), e2 = at(5);
  int64_t E1 = at(6), N1 = at(7), N2 = at(8), E2 = at(9);
  const bool live = s0 < P.nptr4, tlive = T0 < P.nptr4;
  const bool fl = e1 < n1, fr = n2 < e2;  // records far from the leaf on its left, right
  const double rbnd2 = 1. / (P.bound4 * P.bound4);
  const float dvr4f = (float)P.dvr4;
  const float2 dvr4p = make_float2(dvr4f, dvr4f);

  // the tile's nodes: every warp a quarter of the records
  {
    typename std::conditional<Plain, FarSumD, FarSumF>::type s;
    if (tlive) {
      const int first = 32 * warp + lane, step = 32 * kTileLeaves;
      if constexpr (Plain) {
        s.template add<true>(recs, E1, N1, first, step, T0, P.dvr4, rbnd2);
        s.template add<true>(recs, N2, E2, first, step, T0, P.dvr4, rbnd2);
      } else {
        s.template add<true>(recs, E1, N1, first, step, T0, dvr4p);
        s.template add<true>(recs, N2, E2, first, step, T0, dvr4p);
      }
    }
    const double v = s.template total<true>(lane, P.dvr4);
    if (!(lane & 1)) nodeB[warp][lane >> 1] = v;
  }
  const bool tfar = E1 < N1 || N2 < E2;
  // no far range of the tile on a side: the leaf's far range is one
  if (!(E1 < N1)) E1 = N1 = n1;
  if (!(N2 < E2)) N2 = E2 = n2;
  // the leaf's nodes
  {
    typename std::conditional<Plain, FarSumD, FarSumF>::type s;
    if (live) {
      auto range = [&](int64_t i0, int64_t i1) {
        if constexpr (Plain) s.template add<false>(recs, i0, i1, lane, 32, s0, P.dvr4, rbnd2);
        else s.template add<false>(recs, i0, i1, lane, 32, s0, dvr4p);
      };
      if (fl) {
        range(e1, E1);
        range(N1, n1);
      }
      if (fr) {
        range(n2, N2);
        range(E2, e2);
      }
    }
    const double v = s.template total<false>(lane, P.dvr4);
    if (!(lane & 1)) nodeA[warp][lane >> 1] = v;
  }
  // the leaf's points
  typename std::conditional<Plain, double, SumK>::type acc{};
  if (live) {
    auto direct = [&](auto core_c, auto mask_c, int64_t i0, int64_t i1) {
      constexpr bool Core = decltype(core_c)::value, Mask = decltype(mask_c)::value;
      if constexpr (Plain) leaf_direct<Core, Mask>(buf[warp], recs, i0, i1, J, P.dvr4, rbnd2, acc);
      else leaf_direct<Core, Mask>(buf[warp], recs, i0, i1, J, dvr4p, acc);
    };
    const std::true_type yes{};
    const std::false_type no{};
    if (fl) direct(no, yes, lo, e1);  // end inside the leaf: beyond the cores
    const int64_t nl = fl ? n1 : lo, nr = fr ? n2 : hi;
    if (fl && fr) direct(yes, no, nl, nr);
    else direct(yes, yes, nl, nr);
    if (fr) direct(no, yes, e2, hi);
    // mirror records lie below 0 cm-1: none reaches a point past 25 cm-1 (with
    // a step to spare for JMAX's rounding)
    if (nm > 0 && P.v1r4 + P.dvr4 * (double)(s0 - 2) <= P.bound4) direct(yes, yes, n, n + nm);
  }
  __syncthreads();
  Real* R4 = reinterpret_cast<Real*>(a.r4_all) + P.r4_off;
  if (m >= P.nptr4 + 2) return;
  // the reference's R4 is zero past NPTR4 (LBLF4Q :91-94)
  double v = 0.;
  if (m < P.nptr4) {
    if constexpr (Plain) {
      // (far_carry; a tile or leaf without far records has nothing to carry)
      double ref = 0.;
      if (tfar) {
        auto b = [&](int k) { return (nodeB[0][k] + nodeB[1][k]) + (nodeB[2][k] + nodeB[3][k]); };
        const double r = b(kFarRef);
#pragma unroll
        for (int k = 0; k < NP; ++k) v = far_carry(c_farw_plain.tile[k][kLeaf * warp + lane], b(k), r, v);
        ref = r;
      }
      if (fl || fr) {
        const double r = nodeA[warp][kFarRef];
#pragma unroll
        for (int k = 0; k < NP; ++k) v = far_carry(c_farw_plain.leaf[k][lane], nodeA[warp][k], r, v);
        ref += r;
      }
      v = (v + ref) + acc;
    } else {
#pragma unroll
      for (int k = 0; k < NP; ++k) {
        const double b = (nodeB[0][k] + nodeB[1][k]) + (nodeB[2][k] + nodeB[3][k]);
        v = fma(c_farw_mixed.tile[k][kLeaf * warp + lane], b, v);
        v = fma(c_farw_mixed.leaf[k][lane], nodeA[warp][k], v);
      }
      v += acc.value();
    }
  }
  R4[m] = (Real)v;
}

template __global__ void k_f4_far<false>(const __grid_constant__ F4Args);
template __global__ void k_f4_far<true>(const __grid_constant__ F4Args);

}  // namespace clblm
