// jac.cu -- Jacobians of the nadir thermal radiance (noScattJacob,
// clblm_noScattJac.f90:20-339) on the GPU.
//
//   k_interp_map_jobs  (iIn, IP) maps of every layer OD of a block that needs
//                      interpSpectrum's general-ratio branch (the DVout step of
//                      ODLAY, clblm_ODLAY.f90:582-598)
//   k_od_jobs          every layer OD of the block on the uniform grid, binary64
//   k_jac<Plain>       one thread per spectral point: the down-looking
//                      recurrence of Jacobians (:346-716) over the layers,
//                      then the level-temperature derivatives of drv_LevelTemp
//                      (:899-1065) and the molecule derivatives of
//                      drv_LevelConc (:1069-1203)
//
// The per-point recurrence keeps two per-layer arrays in local memory
// (at most kMaxJacLayers layers).  The mixed path runs it in FP32, the FP64
// path in binary64 with the reference's operation order.
#include <cuda_runtime.h>

#include "clblm_common.cuh"
#include "clblm_interpmap.cuh"
#include "clblm_jac.cuh"
#include "clblm_kernels.cuh"
#include "clblm_panel.cuh"
#include "clblm_rt.cuh"

namespace clblm {

// grid (interpolation blocks, jobs); each job its own block list
__global__ void __launch_bounds__(kMapThreads) k_interp_map_jobs(const JacJob* __restrict__ jobs, int njob) {
  const int j = blockIdx.y, b = blockIdx.x;
  if (j >= njob || b >= jobs[j].nblk || !jobs[j].build_map) return;
  const JacJob& jb = jobs[j];
  const int64_t J1 = jb.blk_j1[b];
  if (J1 < 1 || J1 > jb.nout) return;  // a block start off the output grid writes nothing
  interp_map_block(jb.spec.v1, jb.spec.dvin, jb.spec.ratio, J1, jb.blk_vo[b], jb.nout, jb.map);
}

// a product rounded on its own
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// interpSpectrum's linear extension by two points past either end
template <typename Real>
__device__ __forceinline__ Real od_ext_t(const Real* x, int64_t n, int64_t i) {
  if (i >= 1 && i <= n) return x[i - 1];
  if (i == 0 || i == -1) return (Real)2 * x[0] - x[1];
  if (i == n + 1 || i == n + 2) return (Real)2 * x[n - 1] - x[n - 2];
  return (Real)0;
}

// grid (kOdJobPoints-point slices of the longest block, jobs).  A general-
// ratio job reads per point its (iIn, IP) and the 201-point coefficients of
// IP: those four are staged in shared memory, interleaved, since lanes with
// different IP would serialise on the constant cache.
template <bool Plain>
__global__ void __launch_bounds__(kOdJobThreads) k_od_jobs(const JacJob* jobs, int njob, const void* od_all, void* out) {
  using Real = typename std::conditional<Plain, double, float>::type;
  using Real4 = typename std::conditional<Plain, double4, float4>::type;
  __shared__ Real4 ia[203];
  const int j = blockIdx.y;
  if (j >= njob) return;
  const JacJob& jb = jobs[j];
  const int64_t nout = jb.nout;
  const int64_t I0 = (int64_t)blockIdx.x * kOdJobPoints;
  if (I0 >= nout) return;  // the whole CTA, before its barrier
  const Real* x = reinterpret_cast<const Real*>(od_all) + jb.od_off;
  Real* o = reinterpret_cast<Real*>(out) + jb.dst_off;
  const int64_t n_in = jb.n_in;
  const int64_t Iend = min(nout, I0 + kOdJobPoints);
  const bool general = jb.spec.kind != 0 && jb.spec.itype < 0;
  if (general) {  // CTA-uniform
    for (int k = threadIdx.x; k < 203; k += blockDim.x) {
      Real c[4];
      ia_coefs<Real>(k, c);
      ia[k] = {c[0], c[1], c[2], c[3]};
    }
    __syncthreads();
    const int2* map = jb.spec.map;
    for (int64_t I = I0 + threadIdx.x + 1; I <= Iend; I += blockDim.x) {
      const int2 mp = map[I - 1];
      const int64_t i = mp.x;
      const Real4 c = ia[mp.y];
      Real v;
      if (i >= 2 && i + 2 <= n_in) {  // (the extension's tests took most of the kernel)
        const Real* q = x + (i - 2);
        v = fma(c.w, q[3], fma(c.z, q[2], fma(c.y, q[1], mul_rn(c.x, q[0]))));
      } else {
        v = c.x * od_ext_t(x, n_in, i - 1);
        v += c.y * od_ext_t(x, n_in, i);
        v += c.z * od_ext_t(x, n_in, i + 1);
        v += c.w * od_ext_t(x, n_in, i + 2);
      }
      o[I - 1] = v;
    }
    return;
  }
  for (int64_t I = I0 + threadIdx.x + 1; I <= Iend; I += blockDim.x) {
    const Stencil<Real> st = interp_stencil<Real>(jb.spec, I);  // FP32 weights in the mixed path
    Real v = 0;
    if (st.n == 1) v = od_ext_t(x, n_in, st.i[0]);
    else
#pragma unroll
      for (int k = 0; k < 4; ++k) v += st.w[k] * od_ext_t(x, n_in, st.i[k]);
    o[I - 1] = v;
  }
}

template __global__ void k_od_jobs<false>(const JacJob*, int, const void*, void*);
template __global__ void k_od_jobs<true>(const JacJob*, int, const void*, void*);

// ---- the per-point recurrence (Jacobians, down-looking branch) ------------
template <typename Real>
__device__ __forceinline__ Real dev_exp(Real x) {
  if constexpr (sizeof(Real) == 8) return exp(x);
  else return __expf(x);
}

// planckFnDrv, clblm_EMLAY.f90:45-70
template <typename Real>
__device__ __forceinline__ void planck_drv_t(Real V, Real T, Real* B, Real* dB) {
  const Real RC1 = (Real)kRADCN1, RC2 = (Real)kRADCN2;
  Real XKT = T / RC2;
  if (XKT <= (Real)1.e-6) {
    *B = 0;
    *dB = 0;
    return;
  }
  const Real Vr = (Real)V;
  Real cv3 = RC1 * Vr * Vr * Vr;
  Real evt = dev_exp(Vr / XKT);
  *B = cv3 / (evt - 1);
  *dB = *B * *B * (evt * Vr) / (RC2 * cv3 * XKT * XKT);
}

// rlin with its derivative, clblm_EMLAY.f90:187-223
template <typename Real>
__device__ __forceinline__ void rlin_t(Real od, Real* hlf, Real* dhlf) {
  const Real dbAvg2dtau = (Real)(-1. / 12);
  if (od < (Real)1.e-03) {
    *hlf = (Real)0.5 + od * dbAvg2dtau;
    *dhlf = dbAvg2dtau;
  } else if (od > (Real)20.) {
    *hlf = 1 / od;
    *dhlf = -1 / (od * od);
  } else {
    Real tex = dev_exp(od);
    *hlf = 1 / (od)-1 / (tex - 1);
    *dhlf = -1 / (od * od) + tex / ((tex - 1) * (tex - 1));
  }
}

__device__ __forceinline__ double warp_sum_d(double v) {
  // butterfly: every lane ends with the same sum, added in the same order
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

template <bool Plain>
__global__ void __launch_bounds__(128, Plain ? 1 : 8) k_jac(JacArgs a) {
  using Real = typename std::conditional<Plain, double, float>::type;
  int64_t iv = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int N2 = a.nlay;
  constexpr int M = kMaxJacLayers + 2;
  // vector-Jacobian product: per warp, the g-weighted sums of every slot
  const bool vjp = a.g != nullptr;
  __shared__ double s_vjp[kJacMaxWarps][jac_vjp_slots(kMaxJacLayers)];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nslot = jac_vjp_slots(N2);
  if (vjp) {
    for (int k = lane; k < nslot; k += 32) s_vjp[warp][k] = 0.;
    __syncwarp();
  }
  // mixed path: FP32 copies of the profile's per-layer arrays, converted once
  // per block (a conversion from binary64 runs on the FP64 unit)
  enum { kAmf, kTlev, kTlay, kTup, kTlo, kQup, kQlo, kRt100, kNc };
  __shared__ float s_c[Plain ? 1 : kNc][Plain ? 1 : M];
  if constexpr (!Plain) {
    for (int l = threadIdx.x; l <= N2; l += blockDim.x) {
      const bool lay = l < N2;
      auto cv = [&](const double* arr, bool in) { return in && arr ? (float)arr[l] : 0.f; };
      s_c[kTlev][l] = cv(a.tlev, true);
      s_c[kAmf][l] = cv(a.amf_down, lay);
      s_c[kTlay][l] = cv(a.tlay, lay);
      s_c[kTup][l] = cv(a.dT_dTup, lay);
      s_c[kTlo][l] = cv(a.dT_dTlo, lay);
      s_c[kQup][l] = cv(a.dW_dQup, lay);
      s_c[kQlo][l] = cv(a.dW_dQlo, lay);
      s_c[kRt100][l] = lay && a.tlay ? 100.f / (float)a.tlay[l] : 0.f;
    }
    __syncthreads();
  }
  // per-layer value c of layer (or level) i: binary64 on the FP64 path
  auto lc = [&](int c, const double* arr, int i) -> Real {
    if constexpr (Plain) return arr[i];
    else return s_c[c][i];
  };
  // past the block's end: nothing to write; for the product, every lane takes
  // part in the warp sums, with the last point and a zero weight
  const bool live = iv < a.nout;
  if (!live) {
    if (!vjp) return;
    iv = a.nout - 1;
  }
  const double gval = vjp && live ? a.g[a.off + iv] : 0.;
  // one output value: written, or weighted by g and summed over the warp
  auto put = [&](double* dst, int64_t idx, int slot, Real val) {
    if (vjp) {
      const double v = warp_sum_d((double)val * gval);
      if (lane == 0) s_vjp[warp][slot] = v;
    } else if (dst) {
      dst[idx] = (double)val;
    }
  };
  // Of the recurrence's arrays two stay, in local memory: cumTxA, summed from
  // the top and used from the surface, and the down path's dRad_dTau, which
  // first holds cumTxB2 (summed from the surface, used from the top).  The
  // rest is formed again where it is used, an exponential or two each: 13
  // arrays of 62 layers, 3 KB a point, went through L2 and DRAM (8.8 ms of a
  // 60-layer 500 cm-1 call's 85).
  Real cumTxA[M], dTauDn[M];
  const Real* jod = reinterpret_cast<const Real*>(a.jod);
  const double vn = a.v1 + (double)iv * a.dv;
  const Real vr = (Real)vn;  // the point's wavenumber in the working precision, converted once
  // (read-only loads, issued layers ahead: the recurrence is a chain, and a
  // launch of 100,000 points leaves 20 warps an SM to hide 600 cycles a load)
  auto view = [&](int l) -> Real { return __ldg(jod + ((int64_t)(l - 1) * a.nout + iv)); };
  auto variant = [&](int v, int il) -> Real { return __ldg(jod + (((int64_t)v * N2 + il) * a.nout + iv)); };
  auto amf = [&](int l) -> Real { return lc(kAmf, a.amf_down, l - 1); };
  auto down_od = [&](int l, Real od) -> Real { return mul_rn(od, amf(l)); };
  const int lit = a.lin_in_tau;
  const bool dT = a.do_temp != 0;
  auto planck_lev = [&](int lv, Real* B, Real* dB) {  // (levels enter where the source is linear in tau)
    *B = *dB = 0;
    if (lit != 0) planck_drv_t<Real>(vr, lc(kTlev, a.tlev, lv - 1), B, dB);
  };
  auto planck_lay = [&](int l, Real* B, Real* dB) { planck_drv_t<Real>(vr, lc(kTlay, a.tlay, l - 1), B, dB); };
  Real Bsfc, dBsfc;
  planck_drv_t<Real>(vr, (Real)a.tsfc, &Bsfc, &dBsfc);
  Real rad = 0;
  // 0- transmittance along the upwelling path from TOA down
  Real cumODA = 0;
  cumTxA[N2 + 1] = 1;
#pragma unroll 8
  for (int l = N2; l >= 1; --l) {
    cumODA = cumODA + view(l);
    cumTxA[l] = dev_exp(-cumODA);
  }
  const Real totODUp = cumODA, totTxUp = cumTxA[1];
  const bool down = totTxUp > (Real)1.e-06;
  Real dbavgdb, dbavgdbdod, Blt, dTran;
  // 1- downwelling thermal radiance
  if (down) {
    dTauDn[1] = totTxUp;  // cumTxB2
    Real cumODB = 0;
#pragma unroll 8
    for (int l = 1; l <= N2; ++l) {
      cumODB = cumODB + down_od(l, view(l));
      dTauDn[l + 1] = dev_exp(-(totODUp + cumODB));
    }
    Real tx1 = dTauDn[N2 + 1], Bup, dBup;  // of the layer's upper level
    planck_lev(N2 + 1, &Bup, &dBup);
    Real od_next = view(N2);
    for (int l = N2; l >= 1; --l) {
      const Real tx = dTauDn[l], od = down_od(l, od_next);
      od_next = l > 1 ? view(l - 1) : (Real)0;
      dTran = tx - tx1;
      const Real am = amf(l);
      Real B = 0, dB, Blo, dBlo, dtau;
      planck_lev(l, &Blo, &dBlo);
      if (lit != 2) planck_lay(l, &B, &dB);
      if (lit != 0) {
        rlin_t(od, &dbavgdb, &dbavgdbdod);
        if (lit == 2) {
          Blt = Blo + (Bup - Blo) * dbavgdb;
          dtau = (tx1 * Blt - rad + dTran * dbavgdbdod * (Bup - Blo)) * am;
        } else {
          Blt = 2 * B * dbavgdb + Blo * (1 - 2 * dbavgdb);
          dtau = (tx1 * Blt - rad + 2 * dTran * dbavgdbdod * (B - Blo)) * am;
        }
        rad = rad + dTran * Blt;
      } else {
        dtau = (tx1 * B - rad) * am;
        rad = rad + dTran * B;
      }
      dTauDn[l] = dtau;
      tx1 = tx;
      Bup = Blo;
    }
  } else {
    for (int l = 1; l <= N2; ++l) dTauDn[l] = 0;
  }
  // 2- surface reflectance; 3- surface terms
  const Real emis = (Real)a.emis, rsfc = 1 - emis;
  const Real dRad_dEmis = totTxUp * Bsfc - rad;
  const Real dRad_dTsfc = emis * totTxUp * dBsfc;
  rad = rad * rsfc + emis * totTxUp * Bsfc;
  // 5- upwelling thermal radiance, and each layer's derivatives as its level
  // below is complete.
  // drv_LevelTemp: dTau/dT = [tau(T+1) - tau(T)] - (Wtot/T) dTau/dWtot
  // drv_LevelConc: dTau/dln W = the OD of the molecule alone
  // (amfView = 1: the viewing path is the reference path)
  const int64_t o = a.off + iv;
  const bool wantT = dT && (a.dtlev || vjp) && a.vT >= 0, wantM = (a.dqlev || vjp) && a.vM >= 0;
  Real Blo, dBlo, txB = totTxUp, cumODB = 0;  // down path: level l
  planck_lev(1, &Blo, &dBlo);
  Real tx = cumTxA[1];
  Real dTup = 0, dTdn = 0;      // dRad_dT_up(l) and dRad_dT_dn(l) from the layer below
  Real barB = 0;                // dRad_dTbar of the layer below
  Real loT = 0, loM = 0;        // of the layer below at its upper level
  Real m_next = view(1), t_next = wantT ? variant(a.vT, 0) : (Real)0, w_next = wantT ? variant(a.vW, 0) : (Real)0,
       q_next = wantM ? variant(a.vM, 0) : (Real)0;
  for (int l = 1; l <= N2; ++l) {
    const int il = l - 1;
    const Real m = m_next, tp = t_next, wp = w_next, mol = q_next, tx1 = cumTxA[l + 1];
    if (l < N2) {
      m_next = view(l + 1);
      if (wantT) {
        t_next = variant(a.vT, l);
        w_next = variant(a.vW, l);
      }
      if (wantM) q_next = variant(a.vM, l);
    }
    Real Bup, dBup, B = 0, dB = 0;
    planck_lev(l + 1, &Bup, &dBup);
    if (lit != 2) planck_lay(l, &B, &dB);
    // the down path's level and layer temperature terms
    Real dnUp = 0, bar = 0;  // dRad_dT_dn(l + 1) of lit = 2; dRad_dTbar(l)
    if (down && dT) {
      const Real od = down_od(l, m);
      cumODB = cumODB + od;
      const Real txB1 = dev_exp(-(totODUp + cumODB));
      dTran = txB - txB1;
      if (lit != 0) {
        rlin_t(od, &dbavgdb, &dbavgdbdod);
        if (lit == 2) {
          dTdn = dTran * dBlo * (1 - dbavgdb) + dTdn;
          dnUp = dTran * dBup * dbavgdb;
        } else {
          dTdn = dTran * dBlo * (1 - 2 * dbavgdb);
          bar = dTran * 2 * dB * dbavgdb;
        }
      } else {
        bar = dTran * dB;
      }
      txB = txB1;
    }
    Real dtau = dTauDn[l] * rsfc;
    if (dT) bar = bar * rsfc;
    dTran = tx1 - tx;
    Real upUp = 0;  // dRad_dT_up(l + 1)
    if (lit != 0) {
      rlin_t(m, &dbavgdb, &dbavgdbdod);
      if (lit == 2) {
        Blt = Bup * (1 - dbavgdb) + Blo * dbavgdb;
        dtau = dtau + (tx * Blt - rad + dTran * dbavgdbdod * (Blo - Bup));
        if (dT) {
          upUp = dTran * dBup * (1 - dbavgdb);
          dTup = dTup + dTran * dBlo * dbavgdb;
        }
      } else {
        Blt = 2 * B * dbavgdb + Bup * (1 - 2 * dbavgdb);
        dtau = dtau + (tx * Blt - rad + dTran * dbavgdbdod * 2 * (B - Bup));
        if (dT) {
          upUp = dTran * dBup * (1 - 2 * dbavgdb);
          bar = bar + dTran * 2 * dB * dbavgdb;
        }
      }
      rad = rad + dTran * Blt;
    } else {
      dtau = dtau + (tx * B - rad);
      rad = rad + dTran * B;
      if (dT) bar = bar + dTran * dB;
    }
    if (wantT) {
      Real lev = 0;  // dRad_dTlev(l)
      if (lit != 0) lev = dTup + dTdn * rsfc;
      if (lit != 2) {
        lev = lev + bar * lc(kTlo, a.dT_dTlo, il);
        if (l > 1) lev = lev + barB * lc(kTup, a.dT_dTup, il - 1);
        barB = bar;
      }
      Real dTau_dT;
      if constexpr (Plain) {
        dTau_dT = tp - m;
        const double deltaW = 0.01 * a.wtot[il];
        const double dTau_dW = (wp - m) / deltaW;
        const double fac = a.wtot[il] / a.tlay[il];
        dTau_dT = dTau_dT - dTau_dW * fac;
      } else {
        // (wp - m) / (0.01 Wtot) * (Wtot / T) = (wp - m) * 100 / T
        dTau_dT = (tp - m) - (wp - m) * s_c[kRt100][il];
      }
      const Real dRaddT = dtau * dTau_dT;
      const Real up = dRaddT * lc(kTup, a.dT_dTup, il);
      loT = loT + dRaddT * lc(kTlo, a.dT_dTlo, il) + lev;
      put(a.dtlev, (int64_t)il * a.ld + o, il, loT);
      loT = up;
    }
    if (wantM) {
      const Real dRad_dW = dtau * mol;
      const Real up = dRad_dW * lc(kQup, a.dW_dQup, il);
      loM = loM + dRad_dW * lc(kQlo, a.dW_dQlo, il);
      put(a.dqlev, (int64_t)il * a.ld + o, N2 + 1 + il, loM);
      loM = up;
    }
    dTup = upUp;
    dTdn = dnUp;
    tx = tx1;
    Blo = Bup;
    dBlo = dBup;
  }
  if (wantT) {  // the top level
    Real lev = 0;
    if (lit != 0) lev = dTup + dTdn * rsfc;
    if (lit != 2) lev = lev + barB * lc(kTup, a.dT_dTup, N2 - 1);
    put(a.dtlev, (int64_t)N2 * a.ld + o, N2, loT + lev);
  }
  if (wantM) put(a.dqlev, (int64_t)N2 * a.ld + o, 2 * N2 + 1, loM);
  if (a.rad && !vjp) a.rad[o] = (double)rad;
  put(a.dtsfc, o, 2 * N2 + 2, dRad_dTsfc);
  put(a.demis, o, 2 * N2 + 3, dRad_dEmis);
  if (vjp) {  // the CTA's sums, warp by warp in order
    __syncthreads();
    const int nw = (int)(blockDim.x >> 5);
    for (int k = threadIdx.x; k < nslot; k += blockDim.x) {
      double sum = 0.;
      for (int w = 0; w < nw; ++w) sum += s_vjp[w][k];
      a.part[(int64_t)blockIdx.x * nslot + k] = sum;
    }
  }
}

// Sums over the CTAs: a lane per slot, the CTAs dealt to kVjpRows warps, whose
// sums are added in order (one thread per slot waited for 800 loads in turn:
// 114 to 190 us a block)
__global__ void __launch_bounds__(32 * kVjpRows)
    k_vjp_accum(const double* __restrict__ part, int nctas, int nslot, double* __restrict__ acc) {
  __shared__ double rows[kVjpRows][33];
  const int lane = threadIdx.x & 31, row = threadIdx.x >> 5, k = blockIdx.x * 32 + lane;
  double sum = 0.;
  if (k < nslot) {
#pragma unroll 8
    for (int c = row; c < nctas; c += kVjpRows) sum += part[(int64_t)c * nslot + k];
  }
  rows[row][lane] = sum;
  __syncthreads();
  if (row != 0 || k >= nslot) return;
  sum = acc[k];
  for (int w = 0; w < kVjpRows; ++w) sum += rows[w][lane];
  acc[k] = sum;
}

template __global__ void k_jac<false>(JacArgs);
template __global__ void k_jac<true>(JacArgs);

}  // namespace clblm
