// Column phase of one NSW6 step: the column kernel and the saturation
// adjustment (see nsw6_kernels.cu for the step as a whole).
#pragma once

#include <cfloat>
#include <cuda_runtime.h>

#include "nsw6_cell.cuh"
#include "nsw6_common.cuh"
#include "nsw6_fastmath.cuh"

namespace nsw6 {

constexpr int ERR_NOCONV = 3;
constexpr int ERR_NAN = 4;

__device__ __forceinline__ void record_error(DevStatus* st, int code, int k, int g, int l, int iters) {
  if (atomicCAS(&st->code, 0, code) == 0) {
    st->k = k;
    st->g = g;
    st->l = l;
    st->iters = iters;
  }
}

// exp of the column phase: the step's own, or CUDA's (nsw6_set_math).
struct ColumnMath {
  FastMath fm;
  bool lib;
  __device__ __forceinline__ double exp(double x) const { return lib ? soft_slow_exp(x) : fm.exp(x); }
};

// Shared-memory field slots, each [K][COL_TG] doubles.
// S_DQI (the tendency of sedimenting QI) exists in the kernel with the scheme
// switches only.
enum ColSlot {
  S_KINH, S_KINV, S_DRHOE, S_DRHOPHI, S_DKINH, S_DKINV, S_DRHOGU, S_DRHOGV, S_DRHOGW,
  S_DQR, S_DQS, S_DQG, S_RHOF, S_F, S_RHOF2, S_F2, S_VI, S_VJ, S_COUNT,
  S_DQI = S_COUNT, S_COUNT_OPT
};

struct ColumnShared {
  double* f;         // [S_COUNT (S_COUNT_OPT)][K][COL_TG]
  double* grid;      // [GF_COUNT][K]
  double* colacc;    // [6][COL_TG]: precip0, precip1, lh_heat, rhoe, rhophi, rhokin
  int* bmin;         // [2 ntr][K] (room for 8 rows with the switches)
  int* bmax;         // [2 ntr][K]
};

// Which levels of a tile hold anything of a tracer: one bit a level.
constexpr int LEVEL_WORDS = (MAX_KALL + 31) / 32;
__device__ __forceinline__ bool level_bit(const unsigned* m, int k) { return (m[k >> 5] >> (k & 31)) & 1u; }
// any of the levels lo .. hi, or level kc
__device__ __forceinline__ bool any_level(const unsigned* m, int lo, int hi, int kc) {
  if (level_bit(m, kc)) return true;
  for (int w = lo >> 5; w <= hi >> 5; ++w) {
    unsigned x = m[w];
    if (w == lo >> 5) x &= ~0u << (lo & 31);
    if (w == hi >> 5) x &= ~0u >> (31 - (hi & 31));
    if (x) return true;
  }
  return false;
}

// Departure cell of vadv1d_prep for one cell (mod_vadv1d.cpp:355-389).  The
// reference's tmp = k2 * copysign(1, dep - zh(k2)) * copysign(1, zh(k2+1) - dep)
// is k2 when both signs agree and -k2 otherwise; the sign of a difference of
// two doubles is their comparison, so the test is exact integer logic.
//
// The comparisons run on the integer pipe: zk holds cmp_key of the interface
// heights zh, and for non-NaN doubles a >= b exactly when their keys compare
// so; a NaN departure point makes every comparison false, as in the reference.
__device__ __forceinline__ int departure_cell(const double* zh, const long long* zk, int k, double zdis, int bmn,
                                              int bmx, int mkmin, int mkmax) {
  int kc;
  if (bmn == k && bmx == k) {
    kc = k;
  } else {
    kc = 0;
    const double dep = zh[k] - zdis;
    const long long dk = cmp_key(dep);
    const bool nan = is_nan_bits(dep);
    for (int k2 = bmn; k2 <= bmx; ++k2) {
      const bool s1 = !nan && dk >= zk[k2];
      const bool s2 = !nan && zk[k2 + 1] >= dk;
      const int tmp = (s1 == s2) ? k2 : -k2;
      kc = kc > tmp ? kc : tmp;
    }
  }
  if (kc == 0) kc = mkmin;
  if (kc == mkmax + 1) kc = mkmax;
  return kc;
}

// Flux integrals of vadv1d_getflux_new for one cell (mod_vadv1d.cpp:410-449),
// including the small-value filter |f| < EPS -> 0.  In the reference's Kokkos
// lambda the level index is a size_t, so its (k-1)-k2 and k2-k factors are
// evaluated unsigned and never negative; the weight of layer k2 is then
// fact = dz(k2) * 0.25 * ((sign(k2-kc-1)+1) * 2 - 2 * (sign(kc-1-k2)+1)),
// i.e. +dz(k2) above the departure cell, -dz(k2) below it and 0 at it, and
// zdis = zdis0 - fact of the last layer k2 = bmx (flux_rest, the same for every
// flux of a tracer).  Two sources at a time share the weights and keep two
// chains of the FP64 pipe's long latency going.
template <class R>
__device__ __forceinline__ R flux_rest(const R* dz, int k, int kc, R zdis0, int bmn, int bmx) {
  if ((bmn == k && bmx == k) || bmx == kc) return zdis0;
  return zdis0 - (bmx > kc ? dz[bmx] : -dz[bmx]);
}
// |f| >= EPS on the integer pipe (NaN fails, as the comparison does)
__device__ __forceinline__ double flux_filter(double f) {
  const unsigned long long ab = (unsigned long long)__double_as_longlong(f) & 0x7fffffffffffffffull;
  return ab - (unsigned long long)EPS_BITS <= 0x7ff0000000000000ull - (unsigned long long)EPS_BITS ? f : 0.0;
}
__device__ __forceinline__ float flux_filter(float f) { return fabsf(f) >= (float)EPS ? f : 0.0f; }
// n sources src[m] (columns of the tile) into f[m]
template <int TG, int N, class R>
__device__ __forceinline__ void flux_integrals(const R* const (&src)[N], const R* dz, int k, int kc, R rest, int bmn,
                                               int bmx, R (&f)[N]) {
#pragma unroll
  for (int m = 0; m < N; ++m) f[m] = R(0.0);
  if (!(bmn == k && bmx == k)) {
    // the departure cell's own weight is 0 (the reference multiplies by it):
    // adding rhof(kc) * 0 leaves f unchanged and keeps every lane busy
#pragma unroll 1
    for (int k2 = bmn; k2 <= bmx; ++k2) {
      const R w = k2 > kc ? dz[k2] : (k2 < kc ? -dz[k2] : R(0.0));
#pragma unroll
      for (int m = 0; m < N; ++m) f[m] = fmaR(src[m][k2 * TG], w, f[m]);
    }
  }
#pragma unroll
  for (int m = 0; m < N; ++m) f[m] = flux_filter(fmaR(src[m][kc * TG], rest, f[m]));
}

// Kinetic energies of the mixed step (FP32): horizontal, 0.5 |rhog v|^2 / rhog
// of a cell, and vertical, 0.5 rhogw^2 / (c2w0 rhog(k) + c2w1 rhog(k-1)) of a
// half level (mod_precip_transport.cpp:744-766, 991-1011).  The same functions
// form the energies before and after the transport, so a column the transport
// leaves unchanged gets a zero KIN2EIN correction, as in the FP64 step.
__device__ __forceinline__ float kin_h_f(float rvx, float rvy, float rvz, float rhog) {
  return __fdiv_rn(0.5f * __fmaf_rn(rvx, rvx, __fmaf_rn(rvy, rvy, __fmul_rn(rvz, rvz))), rhog);
}
__device__ __forceinline__ float kin_v_f(float rw, float c2w0, float c2w1, float rhog, float rhog_below) {
  return __fdiv_rn(0.5f * __fmul_rn(rw, rw), __fmaf_rn(c2w0, rhog, __fmul_rn(c2w1, rhog_below)));
}

// Newton iteration of the saturation adjustment of one saturated cell:
// satadjust_liq (mod_satadjust.cpp:771-896, the iteration :840-880) or, with
// the switch, satadjust_all (:620-769, the iteration :686-754).  q holds the
// cell's specific humidities with q[QV] = qsum and q[QC] (and q[QI] with
// satadjust_all) = 0; the iteration leaves the adjusted ones there and
// returns the temperature.  Its range, convergence and finiteness tests run
// on the integer pipe (nsw6_fpcmp.cuh).
template <class M>
__device__ __forceinline__ double satadjust_newton(const Problem& P, const Consts& C, const M& mth, bool ice_adj,
                                                   double tem, double ein_moist, double qsum, double rho_l,
                                                   double qd_l, double* q, int k, int g, int l) {
  bool converged = false;
  int ite;
  if (ice_adj) {
    // satadjust_all, mod_satadjust.cpp:686-754 (CPovR = CVovR = 0, all CVW = CVdry)
    const double UL = C.sat_ulimit, LL = C.sat_llimit;
    for (ite = 0; ite < P.itelim; ++ite) {
      const double alpha = dmin(dmax(quo(tem - LL, UL - LL), 0.0), 1.0);
      const double rtem = quo(1.0, fp_max_pos(tem, TEM_MIN));
      const double psatl = PSAT0 * mth.exp(C.LovR_liq * (C.RTEM00 - rtem));
      const double psati = PSAT0 * mth.exp(C.LovR_ice * (C.RTEM00 - rtem));
      const double psat = psatl * alpha + psati * (1.0 - alpha);
      const Divisor by_rt(rho_l * RVAP * tem);
      const double qsatl = soft_div(psatl, by_rt.s, by_rt.b);
      const double qsati = soft_div(psati, by_rt.s, by_rt.b);
      const double qsat = soft_div(psat, by_rt.s, by_rt.b);
      q[I_QV] = qsat;
      q[I_QC] = (qsum - qsat) * alpha;
      q[I_QI] = (qsum - qsat) * (1.0 - alpha);
      double cv = qd_l * CVDRY;
#pragma unroll
      for (int n = 1; n <= 5; ++n) cv = cv + q[n] * CVDRY;
      const double emoist_new = tem * cv + q[I_QV] * LHV0 - q[I_QI] * LHF0;
      const double dalpha_dT = (!(UL - tem < 0.0) && !(tem - LL < 0.0)) ? quo(1.0, UL - LL) : 0.0;
      const double t2 = tem * tem;
      const double dqsatl_dT = quo(C.LovR_liq, t2) * qsatl;
      const double dqsati_dT = quo(C.LovR_ice, t2) * qsati;
      const double dqsat_dT = qsatl * dalpha_dT + dqsatl_dT * alpha - qsati * dalpha_dT + dqsati_dT * (1.0 - alpha);
      const double dqc_dT = (qsum - qsat) * dalpha_dT - dqsat_dT * alpha;
      const double dqi_dT = -(qsum - qsat) * dalpha_dT - dqsat_dT * (1.0 - alpha);
      const double dcv_dT = dqsat_dT * CVDRY + dqc_dT * CVDRY + dqi_dT * CVDRY;
      const double demoist_dT = tem * dcv_dT + cv + dqsat_dT * LHV0 - dqi_dT * LHF0;
      const double dtemp = quo(emoist_new - ein_moist, demoist_dT);
      tem = tem - dtemp;
      if (fp_abs_lt(dtemp, C.dtemp_criteria)) {
        converged = true;
        break;
      }
      if (fp_not_finite(tem)) break;
    }
  } else {
    for (ite = 0; ite < P.itelim; ++ite) {
      const double rtem = quo(1.0, fp_max_pos(tem, TEM_MIN));
      const double psat = PSAT0 * mth.exp(C.LovR_liq * (C.RTEM00 - rtem));
      const double qsat = quo(psat, rho_l * RVAP * tem);
      q[I_QV] = qsat;
      q[I_QC] = qsum - qsat;
      double cv = qd_l * CVDRY;
#pragma unroll
      for (int n = 1; n <= 5; ++n) cv = cv + q[n] * CVDRY;
      const double emoist_new = tem * cv + q[I_QV] * LHV0;
      // dqsat/dT = (LovR/T^2 + CVovR/T) qsat with CVovR = 0, and
      // dCVtot/dT = dqsat/dT (CVW(QV) - CVW(QC)) = 0 (all CVW = CVdry)
      const double dqsat_dT = C.LovR_liq * rtem * rtem * qsat;
      const double demoist_dT = cv + dqsat_dT * LHV0;
      const double dtemp = quo(emoist_new - ein_moist, demoist_dT);
      tem = tem - dtemp;
      if (fp_abs_lt(dtemp, C.dtemp_criteria)) {
        converged = true;
        break;
      }
      if (fp_not_finite(tem)) break;
    }
  }
  if (!converged) record_error(P.status, fp_not_finite(tem) ? ERR_NAN : ERR_NOCONV, k, g, l, ite);
  return tem;
}

// A value loaded here and not sunk to its use: the loads of a pass are in
// flight together before its first call of a soft routine, across which none moves.
__device__ __forceinline__ void loaded(double x) { asm volatile("" ::"d"(x)); }

// The final state of one cell after the transport and KIN2EIN: thermodynamics,
// saturation adjustment, negative filter and outputs (mod_mp_driver.cpp:
// 555-612 with mod_thrmdyn.cpp, mod_satadjust.cpp:274-362 and
// mod_mp_nsw6.cpp:1770-1831) from the cell's rhog and the divisor it makes, rhoge
// (after KIN2EIN), tracers and gsgam2.  With newton = false
// (the column kernel) a saturated interior cell is left as it is and true is
// returned, for nsw6_satadj_kernel; every other cell is finished.  With
// newton = true (that kernel) the cell is saturated: the same values are
// formed, the Newton iteration runs and the cell is finished.
template <class M, bool MIX, bool OPT>
__device__ __forceinline__ bool final_cell(const Problem& P, const Consts& C, const M& mth, bool ice_adj, float lovr_f,
                                           size_t i, size_t iq, size_t KG, bool interior, double rhog,
                                           const Divisor& by_rhog, double rhoge, double (&rq)[6], double gsg,
                                           bool newton, int k, int g, int l) {
  const double rrhog = MIX ? rcp_of(by_rhog) : 0.0;
  double q[6];
#pragma unroll
  for (int n = 0; n < 6; ++n) rq[n] = plus_zero(rq[n]);
  // These quotients must be correctly rounded: the saturation adjustment
  // forms qc = qsum - qsat from them, a difference of nearly equal numbers
  // in which one unit in the last place of qsum is already a relative error
  // of 1e-11 when qc is small.
#pragma unroll
  for (int n = 0; n < 6; ++n) q[n] = MIX ? rq[n] * rrhog : div_rn(rq[n], by_rhog);
  double rho = quo(rhog, gsg);
  const double ein = MIX ? rhoge * rrhog : div_rn(rhoge, by_rhog);
  double qd = 1.0;
#pragma unroll
  for (int n = 1; n <= 5; ++n) qd = qd - q[n];
  // THRMDYN_tempre, mod_thrmdyn.cpp:137-180.  Its temperature is replaced
  // by the saturation adjustment's everywhere and its pressure by the
  // negative filter's at interior levels: only the halo levels output it.
  double pre = 0.0;
  if (!interior) {
    double cvt = 0.0, qdl = 1.0;
#pragma unroll
    for (int n = 1; n <= 5; ++n) {
      cvt = cvt + q[n] * CVDRY;
      qdl = qdl - q[n];
    }
    cvt = cvt + qdl * CVDRY;
    const double tem0 = quo(ein, cvt);
    pre = rho * tem0 * (qdl * RDRY + q[I_QV] * RVAP);
  }

  // SATURATION_adjustment (mod_satadjust.cpp:274-362): ice_adjust = false,
  // or true with the switch (cloud ice joins the adjustment)
  double ein_moist, qsum;
  if (ice_adj) {
    ein_moist = ein + q[I_QV] * LHV0 - q[I_QI] * LHF0;
    qsum = q[I_QV] + q[I_QC] + q[I_QI];
    q[I_QI] = 0.0;
  } else {
    ein_moist = ein + q[I_QV] * LHV0;
    qsum = q[I_QV] + q[I_QC];
  }
  q[I_QV] = qsum;
  q[I_QC] = 0.0;
  // q[QC] (and q[QI] in satadjust_all) is +0 now: its terms leave the sums
  // below as they are (no partial sum is -0), so they are not formed
  // MIX: every CVW is CVdry, so the sum is formed first and scaled once
  double cvtot = MIX ? qd : qd * CVDRY;
#pragma unroll
  for (int n = 2; n <= 5; ++n)
    if (n != I_QI || !ice_adj) cvtot = MIX ? cvtot + q[n] : cvtot + q[n] * CVDRY;
  if (MIX) cvtot = cvtot * CVDRY;
  const double rho_l = rho;
  double tem = quo(ein_moist - q[I_QV] * LHV0, cvtot);
  if (interior) {
    // satadjust_liq (mod_satadjust.cpp:771-896) or satadjust_all
    // (:620-769)
    double qd_l = 1.0;
#pragma unroll
    for (int n = 2; n <= 5; ++n)
      if (n != I_QI || !ice_adj) qd_l = qd_l - q[n];
    if (newton) {
      tem = satadjust_newton(P, C, mth, ice_adj, tem, ein_moist, qsum, rho_l, qd_l, q, k, g, l);
    } else {
    // is the cell saturated?
    // The test qsum - qsat(tem) > EPS is first decided in FP32 (liquid
    // saturation only, sat_screen_liq); the FP64 test decides the rest.
    int sat = ice_adj ? -1 : sat_screen_liq(tem, rho_l, qsum, lovr_f);
    if (sat < 0) {
      const double rtem = quo(1.0, fp_max_pos(tem, TEM_MIN));
      double psat = PSAT0 * mth.exp(C.LovR_liq * (C.RTEM00 - rtem));
      if (ice_adj) {
        const double alpha =
            dmin(dmax(quo(tem - C.sat_llimit, C.sat_ulimit - C.sat_llimit), 0.0), 1.0);
        const double psati = PSAT0 * mth.exp(C.LovR_ice * (C.RTEM00 - rtem));
        psat = psat * alpha + psati * (1.0 - alpha);
      }
      const double qsat = quo(psat, rho_l * RVAP * tem);
      sat = (qsum - qsat > EPS) ? 1 : 0;
    }
    if (sat) return true;
    }
  }
  rq[I_QV] = rhog * q[I_QV];
  rq[I_QC] = rhog * q[I_QC];
  if (ice_adj) rq[I_QI] = rhog * q[I_QI];
  if (!interior) {   // interior levels: rhoge comes from the negative filter below
    soft_branch();
    cvtot = qd * CVDRY;
#pragma unroll
    for (int n = 1; n <= 5; ++n) cvtot = cvtot + q[n] * CVDRY;
    rhoge = rhog * tem * cvtot;
  }

  // negative_filter (mod_mp_nsw6.cpp:1770-1831), interior levels
  double rhog_o = rhog;
  if (interior) {
    double diffq = 0.0;
    unsigned clamped = 0;   // bit n: rq[n] was negative and is now zero
#pragma unroll
    for (int n = 2; n <= 5; ++n) {
      diffq += rq[n];
      if (lt_z(rq[n])) clamped |= 1u << n;
      rq[n] = maxz(rq[n]);
    }
#pragma unroll
    for (int n = 2; n <= 5; ++n) diffq -= rq[n];
    rq[I_QV] += diffq;
    diffq = rq[I_QV];
    rq[I_QV] = maxz(rq[I_QV]);
    diffq -= rq[I_QV];
    double qdf, cva;
    if (fp_is_zero(diffq) && fp_pos_normal(rhog)) {
      // Nothing removed: rhog (1 - diffq) is rhog exactly, and so are
      // rho = rhog / gsg and the reciprocal formed above.  The quotients of
      // the tracers the filter left as they were are those formed above
      // (QR, QS, QG; QI unless the adjustment set it), and an unsaturated
      // cell's cloud water is +0 = (rhog 0) / rhog.
      const unsigned same = (0x34u | (ice_adj && newton ? 0u : 0x08u) | (newton ? 0u : 0x02u)) & ~clamped;
#pragma unroll
      for (int n = 1; n <= 5; ++n)
        if (!((same >> n) & 1u)) q[n] = MIX ? rq[n] * rrhog : div_rn(rq[n], by_rhog);
      // an unsaturated cell's q[QC] (and q[QI] in satadjust_all) is still +0
      const unsigned zero = newton ? 0u : (ice_adj ? 0x0Au : 0x02u);
      qdf = 1.0;
#pragma unroll
      for (int n = 1; n <= 5; ++n)
        if (!((zero >> n) & 1u)) qdf = qdf - q[n];
      cva = CVDRY;   // MIX: qdf CVdry + sum q CVdry is CVdry up to roundings
      if (!MIX) {
        cva = qdf * CVDRY;
#pragma unroll
        for (int n = 1; n <= 5; ++n)
          if (!((zero >> n) & 1u)) cva = cva + q[n] * CVDRY;
      }
    } else {
      rhog_o = rhog * (1.0 - diffq);
      rho = quo(rhog_o, gsg);
      const Divisor by_rhog_o(rhog_o);
      const double rrhog_o = MIX ? rcp_of(by_rhog_o) : 0.0;
#pragma unroll
      for (int n = 1; n <= 5; ++n) q[n] = MIX ? rq[n] * rrhog_o : div_rn(rq[n], by_rhog_o);
      qdf = 1.0;
#pragma unroll
      for (int n = 1; n <= 5; ++n) qdf = qdf - q[n];
      cva = CVDRY;
      if (!MIX) {
        cva = qdf * CVDRY;
#pragma unroll
        for (int n = 1; n <= 5; ++n) cva = cva + q[n] * CVDRY;
      }
    }
    rhoge = tem * rhog_o * cva;
    pre = rho * (qdf * RDRY + q[I_QV] * RVAP) * tem;
  }

  P.rhog[i] = rhog_o;
  P.rhoge[i] = rhoge;
#pragma unroll
  for (int n = 0; n < 6; ++n) {
    P.rhogq[iq + (size_t)n * KG] = rq[n];
    P.q[iq + (size_t)n * KG] = q[n];
  }
  P.rho[i] = rho;
  P.tem[i] = tem;
  P.pre[i] = pre;
  P.qd[i] = qd;
  // mp_driver epilogue (mod_mp_driver.cpp:555-612, MP_DIV_NUM = 1)
  P.re_solid[i] = 20.0E-6;
  P.GDCLW[i] = 0.0;
  P.GDCFRC[i] = 0.0;
  if (!interior) {
    P.GPREC[i] = 0.0;
    P.re_liquid[i] = 0.0;
    P.re_cld[i] = 0.0;
  }
  return false;
}

// MIX: the mixed-precision step: the mass and energy fluxes of the
// sedimentation (mass, internal and potential energy) are integrated and their
// divergences summed in FP64 as in the FP64 step; the kinetic-energy and
// momentum fluxes, their sources, the kinetic energies, their tendencies and
// the KIN2EIN correction are FP32; the quotients of the final state use a
// plain reciprocal and its cv sums are lean (every CVW is CVdry); the state
// updates, the internal-energy budget, the thermodynamics and the saturation
// adjustment stay FP64.
//
// OPT: the kernel with the scheme switches (either precision): QI sedimentation (4
// tracers), the KIN2KIN kinetic-energy correction (mod_precip_transport.cpp:
// 1012-1068) and the mixed-phase saturation adjustment (satadjust_all,
// mod_satadjust.cpp:620-769).
//
// One CTA: COL_TG columns x all levels, NJ cells a thread (cell c of thread t:
// c = t + j blockDim, j < NJ), what only its own thread reads of a cell (its
// mass source, metric factors, departure cells) in registers.  Bound by the
// FP64 pipe and, next to it, by the barriers between a pass that writes a
// level's values and the one that reads its neighbours'.  So the fluxes go in
// pairs (in FP32: threes) that share weights, and the divergence of one pair
// and the sources of the next share a pass: 8 barriers a tracer (5 with the
// FP32 ones) where a pass per flux took 18; and a warp whose levels and those
// they draw on hold nothing of the tracer does none of it (rain above the
// freezing level).  One 16900 x 42 region, FP64: 0.56 -> 0.47 ms (7.1 M -> 6.4 M
// FP64 warp instructions), ten regions in mixed precision
// 5.75 -> 5.18 ms a step.  A pass's loads go first, ahead of the calls of the
// soft routines (no load moves across one, so each would wait for memory by
// itself) and, where registers allow, ahead of the barrier before the pass; the
// final passes take the state from shared memory where their thread has just
// formed it: ten regions 5.11 -> 4.46 ms in mixed precision (a third of whose
// stalls were for memory), 9.35 -> 9.19 ms in FP64.
//
// Threads of a CTA at most, two of which an SM holds (80 registers a thread).
constexpr int COL_THREADS_MAX = 384;

template <int COL_TG, int NJ, bool MIX, bool OPT>
__global__ void __launch_bounds__(COL_THREADS_MAX, 2) nsw6_column_kernel(Problem P, Consts C) {
  extern __shared__ double smraw[];
  const int G = P.gall, K = P.kall, kmin = P.kmin, kmax = P.kmax;
  constexpr int NSLOT = OPT ? S_COUNT_OPT : S_COUNT;
  constexpr int NROW_MAX = OPT ? 8 : 6;
  const int ntr = OPT ? P.ntr : 3;
  const int nrow = 2 * ntr;
  const bool kin2kin = OPT && C.opt_kin2kin != 0.0;
  const bool ice_adj = OPT && C.opt_expice == 0.0;
  const int l = blockIdx.y;
  const int g0 = blockIdx.x * COL_TG;
  const size_t KG = (size_t)K * G;
  const size_t off = (size_t)l * KG;
  const size_t offq = (size_t)l * NQ * KG;
  const int ncell = K * COL_TG;
  const double dt = P.dt;

  ColumnShared S;
  S.f = smraw;
  S.grid = S.f + (size_t)NSLOT * ncell;
  S.colacc = S.grid + GF_COUNT * K;
  long long* zkey = reinterpret_cast<long long*>(S.colacc + 6 * COL_TG);   // [2][K]: cmp_key of gzh, gzshift
  S.bmin = reinterpret_cast<int*>(zkey + 2 * K);
  S.bmax = S.bmin + NROW_MAX * K;
  // MIX: dgz, dgzh, rdgz, rdgzh, afact, bfact, cfact, dfact in FP32
  float* gf = reinterpret_cast<float*>(S.bmax + NROW_MAX * K);
  __shared__ unsigned held[8][LEVEL_WORDS];   // levels with a source, per tracer on full and half levels
  auto F = [&](int slot) { return S.f + (size_t)slot * ncell; };
  // FP32 views of slots (MIX): a slot's FP32 view has two halves, [0, ncell)
  // and [ncell, 2 ncell); the thread of cell c owns entries c and ncell + c.
  auto FF = [&](int slot) { return reinterpret_cast<float*>(S.f + (size_t)slot * ncell); };

  for (int c = threadIdx.x; c < GF_COUNT * K; c += blockDim.x) S.grid[c] = P.grid[c];
  for (int c = threadIdx.x; c < 2 * K; c += blockDim.x)
    zkey[c] = cmp_key(P.grid[(c < K ? GF_GZH : GF_GZSHIFT) * K + c % K]);
  for (int c = threadIdx.x; c < 8 * LEVEL_WORDS; c += blockDim.x) held[c / LEVEL_WORDS][c % LEVEL_WORDS] = 0u;
  // MIX: the tile's unit vectors ix, iy, iz, jx, jy, jz in FP32 ([6][COL_TG]);
  // they meet FP32 values only (the velocity components, the momentum tendencies)
  float* uvf = gf + 8 * K;
  if (MIX) {
    const int rows[8] = {GF_DGZ, GF_DGZH, GF_RDGZ, GF_RDGZH, GF_AFACT, GF_BFACT, GF_CFACT, GF_DFACT};
    for (int c = threadIdx.x; c < 8 * K; c += blockDim.x) gf[c] = (float)P.grid[rows[c / K] * K + c % K];
    for (int c = threadIdx.x; c < 6 * COL_TG; c += blockDim.x) {
      const int a = c / COL_TG, g = g0 + c % COL_TG;
      const double* u = a == 0 ? P.ix : a == 1 ? P.iy : a == 2 ? P.iz : a == 3 ? P.jx : a == 4 ? P.jy : P.jz;
      uvf[c] = g < G ? (float)u[(size_t)l * G + g] : 0.0f;
    }
  }
  for (int c = threadIdx.x; c < 6 * COL_TG; c += blockDim.x) S.colacc[c] = 0.0;
  __syncthreads();
  const ColumnMath mth{FastMath(P.fmtab), P.math_lib != 0};   // (few cells ask for it: tables through L1)
  const double* gzh = S.grid + GF_GZH * K;
  const double* gzs = S.grid + GF_GZSHIFT * K;
  const double* dgz = S.grid + GF_DGZ * K;
  const double* dgzh = S.grid + GF_DGZH * K;
  const double* rdgz = S.grid + GF_RDGZ * K;
  const double* rdgzh = S.grid + GF_RDGZH * K;
  const double* afact = S.grid + GF_AFACT * K;
  const double* bfact = S.grid + GF_BFACT * K;
  const double* cfact = S.grid + GF_CFACT * K;
  const double* dfact = S.grid + GF_DFACT * K;

  // ---- kcell_min/max per level from the region extrema (mod_vadv1d.cpp:316-353)
  for (int c = threadIdx.x; c < nrow * K; c += blockDim.x) {
    const int s = c / K, k = c % K;
    const int half = s / ntr;
    const int mkmin = half ? kmin + 1 : kmin;
    const double* zh = half ? gzs : gzh;
    int bmn = k, bmx = k;
    if (k >= mkmin && k <= kmax) {
      const size_t e = ((size_t)l * nrow + s) * K + k;
      const unsigned long long kx = P.zmax[e], kn = P.zmin[e];
      double zzmax = DBL_MIN, zzmin = DBL_MIN;
      if (kx != 0ull) {
        const double v = key_value(kx);
        zzmax = v > zzmax ? v : zzmax;
      }
      if (kn != ~0ull) {
        const double v = key_value(kn);
        zzmin = v < zzmin ? v : zzmin;
      }
      if (zzmax > 0.0) {
        for (int k2 = k; k2 >= mkmin; --k2)
          if ((zh[k2] <= zh[k] - zzmax) && (zh[k2 + 1] > zh[k] - zzmax)) {
            bmn = k2;
            break;
          }
      }
      if (zzmin < 0.0) {
        for (int k2 = k; k2 <= kmax; ++k2)
          if ((zh[k2] <= zh[k] - zzmin) && (zh[k2 + 1] > zh[k] - zzmin)) {
            bmx = k2;
            break;
          }
      }
    }
    S.bmin[c] = bmn;
    S.bmax[c] = bmx;
  }

  // A thread's own values of its cells, in registers across the passes.
  double r_rgs[NJ];                            // gam2 / gsgam2
  double r_rgsh[NJ], r_c2w0[NJ], r_c2w1[NJ];   // gam2h / gsgam2h and C2Wfact at half level k
  // MIX: gam2h / gsgam2h (it scales FP32 sources only) and C2Wfact (they
  // scale the FP32 vertical kinetic energies only) in FP32
  float r_rgshf[NJ], r_c2w0f[NJ], r_c2w1f[NJ];
  const float* dgzf = gf;
  const float* dgzhf = gf + K;
  const float* rdgzf = gf + 2 * K;
  const float* rdgzhf = gf + 3 * K;
  const float* aff = gf + 4 * K;   // MIX: afact, bfact, cfact, dfact in FP32
  const float* bff = gf + 5 * K;
  const float* cff = gf + 6 * K;
  const float* dff = gf + 7 * K;
  // Bit j (8 + j): a factor of the cell's sources (of its half level's) is an
  // infinity or a NaN, which a zero mass does not make a zero: the products are
  // formed all the same, and a NaN flux is filtered out.  (A level with nothing
  // else adds nothing to a flux, so the levels held and `act` leave it out.)
  unsigned odd = 0;
  auto infinite = [](float x) { return (soft_float_bits(x) & 0x7F800000u) == 0x7F800000u; };

  // ---- metric factors, kinetic energy, zeroed accumulators
  //      (mod_precip_transport.cpp:715-770, cnvvar_rhogkin_in mod_debug.cpp:269-330)
  // MIX keeps these FP32 values in the FP32 halves of slots it uses as FP32:
  //   S_KINH: kinetic energy (horizontal) | rhog (before, then after the transport)
  //   S_KINV: kinetic energy (vertical)   | gam2 / gsgam2 of the cell
  //   S_DKINH: its tendency               |
  //   S_DKINV: its tendency               | rhogw of the half level (before)
  //   S_VI, S_VJ: the velocity components | gsgam2h, gsgam2 of the cell
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int c = threadIdx.x + j * blockDim.x;
    r_rgs[j] = r_rgsh[j] = r_c2w0[j] = r_c2w1[j] = 0.0;
    r_rgshf[j] = r_c2w0f[j] = r_c2w1f[j] = 0.0f;
    if (c >= ncell) continue;
    for (int s = S_KINH; s <= S_DQG; ++s) F(s)[c] = 0.0;   // (a slot's two FP32 halves are zero as well)
    if (OPT) F(S_DQI)[c] = 0.0;
    F(S_VI)[c] = 0.0;
    F(S_VJ)[c] = 0.0;
  }
  if (MIX) __syncthreads();   // a slot's halves belong to other threads than its doubles
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int c = threadIdx.x + j * blockDim.x;
    if (c >= ncell) continue;
    const int k = c / COL_TG, gx = c % COL_TG, g = g0 + gx;
    if (g >= G) continue;
    const size_t i = off + (size_t)k * G + g;
    const size_t ic = (size_t)l * G + g;
    const bool interior = (k >= kmin && k <= kmax);
    const double gsg = P.gsgam2[i], gm = P.gam2[i], gsh = P.gsgam2h[i], gmh = P.gam2h[i], rg = P.rhog[i];
    const double vxd = P.vx[i], vyd = P.vy[i], vzd = P.vz[i];
    const double rvx = P.rhogvx[i], rvy = P.rhogvy[i], rvz = P.rhogvz[i], rwd = MIX ? P.rhogw[i] : 0.0;
    loaded(gsg), loaded(gm), loaded(gsh), loaded(gmh), loaded(rg), loaded(vxd), loaded(vyd), loaded(vzd);
    loaded(rvx), loaded(rvy), loaded(rvz);
    if (MIX) loaded(rwd);
    // gam2 / gsgam2 and afact / gsgam2, correctly rounded
    const Divisor by_gsg(gsg);
    if (interior) r_rgs[j] = div_rn(gm, by_gsg);
    if (MIX) {
      // the velocity components scale FP32 momentum sources only: FP32
      const float vx = soft_d2f(vxd), vy = soft_d2f(vyd), vz = soft_d2f(vzd);
      const float vi = __fmaf_rn(vz, uvf[2 * COL_TG + gx], __fmaf_rn(vy, uvf[1 * COL_TG + gx], __fmul_rn(vx, uvf[gx])));
      const float vj =
          __fmaf_rn(vz, uvf[5 * COL_TG + gx], __fmaf_rn(vy, uvf[4 * COL_TG + gx], __fmul_rn(vx, uvf[3 * COL_TG + gx])));
      float rgs = 0.0f, kin = 0.0f;
      FF(S_VI)[c] = vi;
      FF(S_VJ)[c] = vj;
      const float gsgf = soft_d2f(gsg), ghf = soft_d2f(gsh), rhogf = soft_d2f(rg);
      FF(S_VI)[ncell + c] = ghf;
      FF(S_VJ)[ncell + c] = gsgf;
      FF(S_KINH)[ncell + c] = rhogf;
      if (interior) {
        FF(S_KINV)[ncell + c] = rgs = soft_d2f(r_rgs[j]);
        FF(S_KINH)[c] = kin = kin_h_f(soft_d2f(rvx), soft_d2f(rvy), soft_d2f(rvz), rhogf);
      }
      if (k >= kmin + 1 && k <= kmax) {
        r_c2w0f[j] = __fmul_rn(__fdiv_rn(aff[k], gsgf), ghf);
        r_rgshf[j] = __fdiv_rn(soft_d2f(gmh), ghf);
        FF(S_DKINV)[ncell + c] = soft_d2f(rwd);
      }
      if (infinite(vi) || infinite(vj) || infinite(rgs) || infinite(kin)) odd |= 1u << j;
      continue;
    }
    const double vi = vxd * P.ix[ic] + vyd * P.iy[ic] + vzd * P.iz[ic];
    const double vj = vxd * P.jx[ic] + vyd * P.jy[ic] + vzd * P.jz[ic];
    F(S_VI)[c] = vi;
    F(S_VJ)[c] = vj;
    double kin = 0.0;
    if (interior) F(S_KINH)[c] = kin = quo(0.5 * (rvx * rvx + rvy * rvy + rvz * rvz), rg);
    if (fp_not_finite(vi) || fp_not_finite(vj) || fp_not_finite(r_rgs[j]) || fp_not_finite(kin)) odd |= 1u << j;
    if (k >= kmin + 1 && k <= kmax) {
      r_c2w0[j] = div_rn(afact[k], by_gsg) * gsh;
      r_rgsh[j] = quo(gmh, gsh);
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int c = threadIdx.x + j * blockDim.x;
    if (c >= ncell) continue;
    const int k = c / COL_TG, g = g0 + c % COL_TG;
    if (g >= G || k < kmin + 1 || k > kmax) continue;
    const size_t i = off + (size_t)k * G + g;
    if (MIX) {
      const float c2w1 = __fmul_rn(__fdiv_rn(bff[k], FF(S_VJ)[ncell + c - COL_TG]), FF(S_VI)[ncell + c]);
      const float rw = FF(S_DKINV)[ncell + c];
      const float kin = kin_v_f(rw, r_c2w0f[j], c2w1, FF(S_KINH)[ncell + c], FF(S_KINH)[ncell + c - COL_TG]);
      FF(S_KINV)[c] = kin;
      if (infinite(kin) || infinite(r_rgshf[j])) odd |= 0x100u << j;   // (an infinite rw gives no finite kin)
      r_c2w1f[j] = c2w1;
      continue;
    }
    const double c2w0 = r_c2w0[j];
    const double gsgm = P.gsgam2[i - G], gsh = P.gsgam2h[i], rw = P.rhogw[i], rg = P.rhog[i], rgm = P.rhog[i - G];
    loaded(gsgm), loaded(gsh), loaded(rw), loaded(rg), loaded(rgm);
    const double c2w1 = div_rn(bfact[k], Divisor(gsgm)) * gsh;
    const double kin = quo(0.5 * (rw * rw), c2w0 * rg + c2w1 * rgm);
    F(S_KINV)[c] = kin;
    if (fp_not_finite(kin) || fp_not_finite(r_rgsh[j])) odd |= 0x100u << j;   // (an infinite rw gives no finite kin)
    r_c2w1[j] = c2w1;
  }
  // (the vertical kinetic energies are next read by their own threads, after barriers by others)

  // ---- sedimentation of QR, QS, QG (mod_precip_transport.cpp:767-955)
  // tracers in the reference's order (QI sediments with "4WATER")
  double bq[NJ];        // rhoq = rhogq gam2 / gsgam2 of the cell; then, FP64, qh of the half level
  double rest[NJ];      // flux_rest of the cell
  float restf[NJ];      // MIX: in FP32
  int kc[NJ];           // departure cell
  // notes the levels whose cells of the tile hold something (a warp's lanes at a time)
  auto note = [&](unsigned* m, int c, bool holds) {
    const unsigned b = __ballot_sync(0xffffffffu, holds);
    const int lane = threadIdx.x & 31;
    constexpr unsigned group = COL_TG >= 32 ? 0xffffffffu : (1u << COL_TG) - 1u;
    if (lane % COL_TG == 0 && ((b >> lane) & group)) {
      const int k = c / COL_TG;
      atomicOr(&m[k >> 5], 1u << (k & 31));
    }
  };
  for (int t = 0; t < ntr; ++t) {
    const int nq = ntr == 4 ? (t == 0 ? I_QR : t == 1 ? I_QI : t == 2 ? I_QS : I_QG) : (t == 0 ? I_QR : t == 1 ? I_QS : I_QG);
    const int dqs_slot = nq == I_QR ? S_DQR : nq == I_QS ? S_DQS : nq == I_QG ? S_DQG : S_DQI;
    // departure distances of this region: [2 ntr][K][G] rows t (full) and ntr + t (half)
    const double* zdis0 = P.zdis + ((size_t)l * nrow + t) * KG;
    const double* zdis0h = P.zdis + ((size_t)l * nrow + ntr + t) * KG;
    const int* bmn_f = S.bmin + t * K;
    const int* bmx_f = S.bmax + t * K;
    const int* bmn_h = S.bmin + (ntr + t) * K;
    const int* bmx_h = S.bmax + (ntr + t) * K;
    const double* rhogq_n = P.rhogq + offq + (size_t)nq * KG;
    const double* q_n = P.q + offq + (size_t)nq * KG;
    unsigned act = 0;   // bit j: the cell draws on levels that hold something
    double ld0[NJ], ld1[NJ], ld2[NJ], ld3[NJ];   // a pass's loads
    // loads of the half levels' pass: departure distance, q of the two levels (and rhogw)
    auto load_half = [&]() {
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int c = threadIdx.x + j * blockDim.x;
        const int k = c / COL_TG, g = g0 + c % COL_TG;
        if (c >= ncell || g >= G || k < kmin + 1 || k > kmax) continue;
        const size_t i = (size_t)k * G + g;
        ld0[j] = zdis0h[i];
        ld1[j] = q_n[i];
        ld2[j] = q_n[i - G];
        if (!MIX) ld3[j] = P.rhogw[off + i];
        loaded(ld0[j]), loaded(ld1[j]), loaded(ld2[j]);
        if (!MIX) loaded(ld3[j]);
      }
    };

    // departure cells (full levels), rhoq = rhogq * rgs, which is the source of
    // the first flux (the mass flux), and the source of the second (energy)
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int c = threadIdx.x + j * blockDim.x;
      const int k = c / COL_TG, g = g0 + c % COL_TG;
      if (c >= ncell || g >= G) continue;
      const size_t i = (size_t)k * G + g;
      ld0[j] = rhogq_n[i];
      ld1[j] = zdis0[i];
      ld2[j] = P.tem[off + i];
      loaded(ld0[j]), loaded(ld1[j]), loaded(ld2[j]);
    }
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int c = threadIdx.x + j * blockDim.x;
      const int k = c / COL_TG, gx = c % COL_TG, g = g0 + gx;
      bq[j] = 0.0;
      rest[j] = 0.0;
      restf[j] = 0.0f;
      kc[j] = kmin;
      const bool own = c < ncell && g < G;
      if (own) {
        const double b0 = ld0[j];
        if (fp_not_finite(ld2[j])) odd |= 1u << j;
        if (!fp_is_zero(b0) || ((odd >> j) & 1u)) {
          soft_branch();
          bq[j] = b0 * r_rgs[j];
        }
        if (k >= kmin && k <= kmax) {
          const double z = ld1[j];
          kc[j] = departure_cell(gzh, zkey, k, z, bmn_f[k], bmx_f[k], kmin, kmax);
          rest[j] = flux_rest(dgz, k, kc[j], z, bmn_f[k], bmx_f[k]);
          if (MIX) restf[j] = flux_rest(dgzf, k, kc[j], soft_d2f(z), bmn_f[k], bmx_f[k]);
        }
      }
      const double b = bq[j];
      const bool holds = own && !fp_is_zero(b);
      if (c < ncell) {
        double e = 0.0;
        if (holds || ((odd >> j) & 1u)) {
          soft_branch();
          e = b * CVDRY * ld2[j];
        }
        F(S_RHOF)[c] = b;
        F(S_RHOF2)[c] = e;
      }
      note(held[t], c, holds);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int c = threadIdx.x + j * blockDim.x;
      const int k = c / COL_TG;
      if (c < ncell && g0 + c % COL_TG < G && k >= kmin && k <= kmax && any_level(held[t], bmn_f[k], bmx_f[k], kc[j]))
        act |= 1u << j;
    }

    // sources 2 .. 5 (mod_precip_transport.cpp:776-808): potential energy (of the cell's z),
    // horizontal kinetic energy, momentum along i and j
    auto source = [&](int f, int c, int j, double z) {
      const double b = bq[j];
      if (fp_is_zero(b) && !((odd >> j) & 1u)) return 0.0;
      soft_branch();
      switch (f) {
        case 2: return b * GRAV * z;
        case 4: return b * F(S_VI)[c];
        default: return b * F(S_VJ)[c];
      }
    };
    // flux divergence and surface fluxes (mod_precip_transport.cpp:782-842,
    // 900-954)
    auto divergence = [&](int f, int c, const double* fl) {
      const int k = c / COL_TG, gx = c % COL_TG, g = g0 + gx;
      if (g >= G || k < kmin || k > kmax) return;
      const double fk = fl[c], fk1 = fl[c + COL_TG];
      const bool none = fp_is_zero(fk) && fp_is_zero(fk1);
      double d = 0.0;
      const int s = f == 1 ? S_DRHOE : f == 2 ? S_DRHOPHI : f == 3 ? S_DKINH : f == 4 ? S_DRHOGU : S_DRHOGV;
      if (!none) {
        soft_branch();
        d = (fk1 - fk) * rdgz[k];
        if (f != 0) F(s)[c] = F(s)[c] - d;
      }
      if (f == 0) {
        F(dqs_slot)[c] = none ? 0.0 : -d;
        if (nq == I_QR) P.GPREC[off + (size_t)k * G + g] = fp_is_zero(fk) ? 0.0 : soft_div_rn(-fk, P.by_dt, dt);
      }
      if (k == kmin && !fp_is_zero(fk)) {
        double* acc = S.colacc;
        const double fdt = soft_div_rn(fk, P.by_dt, dt);
        switch (f) {
          case 0:
            if (nq == I_QR) {
              acc[0 * COL_TG + gx] = acc[0 * COL_TG + gx] - fdt;
            } else {
              acc[1 * COL_TG + gx] = acc[1 * COL_TG + gx] - fdt;
              acc[2 * COL_TG + gx] = acc[2 * COL_TG + gx] + soft_div_rn(fk * LHF0, P.by_dt, dt);
            }
            break;
          case 1: acc[3 * COL_TG + gx] = acc[3 * COL_TG + gx] - fdt; break;
          case 2: acc[4 * COL_TG + gx] = acc[4 * COL_TG + gx] - fdt; break;
          case 3: acc[5 * COL_TG + gx] = acc[5 * COL_TG + gx] - fdt; break;
          default: break;
        }
      }
    };
    // two FP64 fluxes of every cell, S_RHOF into S_F and S_RHOF2 into S_F2
    auto flux_pair = [&](bool half) {
      const double* dz = half ? dgzh : dgz;
      const int* bmn = half ? bmn_h : bmn_f;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int c = threadIdx.x + j * blockDim.x;
        if (c >= ncell) continue;
        const int k = c / COL_TG, gx = c % COL_TG;
        double fl[2] = {0.0, 0.0};
        if ((act >> j) & 1u) {
          soft_branch();
          const double* const src[2] = {F(S_RHOF) + gx, F(S_RHOF2) + gx};
          // (the reference passes the full levels' upper bound to the half levels too)
          flux_integrals<COL_TG, 2>(src, dz, k, kc[j], rest[j], bmn[k], bmx_f[k], fl);
        }
        F(S_F)[c] = fl[0];
        F(S_F2)[c] = fl[1];
      }
    };
    // half levels: departure cells, qh and the sources of the two half-level
    // fluxes (mod_precip_transport.cpp:845-882)
    auto half_sources = [&](int j) {
      const int c = threadIdx.x + j * blockDim.x;
      const int k = c / COL_TG, gx = c % COL_TG, g = g0 + gx;
      const bool hv = c < ncell && g < G && k >= kmin + 1 && k <= kmax;
      double qs = 0.0;
      if (hv) {
        const double z = ld0[j];
        kc[j] = departure_cell(gzs, zkey + K, k, z, bmn_h[k], bmx_h[k], kmin + 1, kmax);
        if (MIX) restf[j] = flux_rest(dgzhf, k, kc[j], soft_d2f(z), bmn_h[k], bmx_f[k]);
        else rest[j] = flux_rest(dgzh, k, kc[j], z, bmn_h[k], bmx_f[k]);
        const double qa = ld1[j], qb = ld2[j];
        const bool some = !(fp_is_zero(qa) && fp_is_zero(qb)), full = some || ((odd >> (8 + j)) & 1u);
        if (MIX) {
          // qh scales the FP32 sources of the two half-level fluxes only: FP32
          const float qh = full ? 0.5f * (soft_d2f(qa) + soft_d2f(qb)) * r_rgshf[j] : 0.0f;
          FF(S_RHOF)[c] = __fmul_rn(qh, FF(S_KINV)[c]);
          FF(S_RHOF)[ncell + c] = __fmul_rn(qh, FF(S_DKINV)[ncell + c]);   // rhogw before the transport
        } else {
          double s0 = 0.0, s1 = 0.0;
          if (full) {
            soft_branch();
            const double qh = 0.5 * (qa + qb) * r_rgsh[j];
            s0 = qh * F(S_KINV)[c];
            s1 = qh * ld3[j];
          }
          F(S_RHOF)[c] = s0;
          F(S_RHOF2)[c] = s1;
        }
        qs = some ? 1.0 : 0.0;
      } else if (c < ncell) {
        if (MIX) {
          FF(S_RHOF)[c] = FF(S_RHOF)[ncell + c] = 0.0f;
        } else {
          F(S_RHOF)[c] = 0.0;
          F(S_RHOF2)[c] = 0.0;
        }
      }
      note(held[ntr + t], c, qs != 0.0);
    };
    auto half_active = [&]() {
      act = 0;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int c = threadIdx.x + j * blockDim.x;
        const int k = c / COL_TG;
        if (c < ncell && g0 + c % COL_TG < G && k >= kmin + 1 && k <= kmax &&
            any_level(held[ntr + t], bmn_h[k], max(bmx_f[k], bmn_h[k]), kc[j]))
          act |= 1u << j;
      }
    };

    flux_pair(false);   // mass and internal energy
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int c = threadIdx.x + j * blockDim.x;
      const int k = c / COL_TG, g = g0 + c % COL_TG;
      if (c >= ncell || g >= G) continue;
      const size_t i = (size_t)k * G + g;
      ld0[j] = P.z[off + i];
      ld1[j] = q_n[i];
      loaded(ld0[j]), loaded(ld1[j]);
      if (fp_not_finite(ld0[j])) odd |= 1u << j;
    }
    __syncthreads();
    if (!MIX) {
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int c = threadIdx.x + j * blockDim.x;
        if (c >= ncell) continue;
        divergence(0, c, F(S_F));
        divergence(1, c, F(S_F2));
        F(S_RHOF)[c] = source(2, c, j, ld0[j]);
        double e = 0.0;
        if (!fp_is_zero(bq[j]) || ((odd >> j) & 1u)) {
          soft_branch();
          e = ld1[j] * r_rgs[j] * F(S_KINH)[c];
        }
        F(S_RHOF2)[c] = e;
      }
      __syncthreads();
      flux_pair(false);   // potential and horizontal kinetic energy
      __syncthreads();
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int c = threadIdx.x + j * blockDim.x;
        if (c >= ncell) continue;
        divergence(2, c, F(S_F));
        divergence(3, c, F(S_F2));
        F(S_RHOF)[c] = source(4, c, j, 0.0);
        F(S_RHOF2)[c] = source(5, c, j, 0.0);
      }
      __syncthreads();
      flux_pair(false);   // momentum along i and j
      load_half();
      __syncthreads();
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int c = threadIdx.x + j * blockDim.x;
        if (c < ncell) {
          divergence(4, c, F(S_F));
          divergence(5, c, F(S_F2));
        }
        half_sources(j);
      }
      __syncthreads();
      half_active();
      flux_pair(true);    // vertical kinetic energy and momentum w
      __syncthreads();
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int c = threadIdx.x + j * blockDim.x;
        const int k = c / COL_TG, g = g0 + c % COL_TG;
        if (c >= ncell || g >= G || k < kmin + 1 || k > kmax) continue;
        const double a1 = F(S_F)[c], a0 = F(S_F)[c - COL_TG], b1 = F(S_F2)[c], b0 = F(S_F2)[c - COL_TG];
        if (!(fp_is_zero(a1) && fp_is_zero(a0) && fp_is_zero(b1) && fp_is_zero(b0))) {
          soft_branch();
          F(S_DKINV)[c] = F(S_DKINV)[c] - (a1 - a0) * rdgzh[k];
          F(S_DRHOGW)[c] = F(S_DRHOGW)[c] - (b1 - b0) * rdgzh[k];
        }
      }
      continue;   // the next tracer's sources go to S_RHOF, which nobody reads now
    }
    // MIX: the mass and energy fluxes (mass, internal and potential energy) as
    // in the FP64 step; the kinetic-energy and momentum ones, their sources and
    // tendencies in FP32, in the halves of S_RHOF2 and S_F2 and the free upper
    // ones of the FP32 accumulators
    float* const srcf[3] = {FF(S_RHOF2), FF(S_RHOF2) + ncell, FF(S_DRHOGU) + ncell};
    float* const fluxf[3] = {FF(S_F2), FF(S_F2) + ncell, FF(S_DRHOGV) + ncell};
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int c = threadIdx.x + j * blockDim.x;
      if (c >= ncell) continue;
      divergence(0, c, F(S_F));
      divergence(1, c, F(S_F2));
      F(S_RHOF)[c] = source(2, c, j, ld0[j]);
      // (S_RHOF2's doubles were read before the last barrier)
      float r3 = 0.0f, r4 = 0.0f, r5 = 0.0f;
      if (!fp_is_zero(bq[j]) || ((odd >> j) & 1u)) {
        const float bf = soft_d2f(bq[j]);
        r3 = __fmul_rn(__fmul_rn(soft_d2f(ld1[j]), FF(S_KINV)[ncell + c]), FF(S_KINH)[c]);
        r4 = __fmul_rn(bf, FF(S_VI)[c]);
        r5 = __fmul_rn(bf, FF(S_VJ)[c]);
      }
      srcf[0][c] = r3;
      srcf[1][c] = r4;
      srcf[2][c] = r5;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int c = threadIdx.x + j * blockDim.x;
      if (c >= ncell) continue;
      const int k = c / COL_TG, gx = c % COL_TG;
      double fl[1] = {0.0};
      float ff[3] = {0.0f, 0.0f, 0.0f};
      if ((act >> j) & 1u) {
        const double* const src[1] = {F(S_RHOF) + gx};
        flux_integrals<COL_TG, 1>(src, dgz, k, kc[j], rest[j], bmn_f[k], bmx_f[k], fl);
        const float* const sf[3] = {srcf[0] + gx, srcf[1] + gx, srcf[2] + gx};
        flux_integrals<COL_TG, 3>(sf, dgzf, k, kc[j], restf[j], bmn_f[k], bmx_f[k], ff);
      }
      F(S_F)[c] = fl[0];
      fluxf[0][c] = ff[0];
      fluxf[1][c] = ff[1];
      fluxf[2][c] = ff[2];
    }
    load_half();
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int c = threadIdx.x + j * blockDim.x;
      const int k = c / COL_TG, gx = c % COL_TG, g = g0 + gx;
      if (c < ncell) {
        divergence(2, c, F(S_F));
        if (g < G && k >= kmin && k <= kmax) {
          FF(S_DKINH)[c] = FF(S_DKINH)[c] - (fluxf[0][c + COL_TG] - fluxf[0][c]) * rdgzf[k];
          FF(S_DRHOGU)[c] = FF(S_DRHOGU)[c] - (fluxf[1][c + COL_TG] - fluxf[1][c]) * rdgzf[k];
          FF(S_DRHOGV)[c] = FF(S_DRHOGV)[c] - (fluxf[2][c + COL_TG] - fluxf[2][c]) * rdgzf[k];
          // the kinetic energy reaching the ground (precip_rhokin)
          if (k == kmin && fluxf[0][c] != 0.0f)
            S.colacc[5 * COL_TG + gx] = S.colacc[5 * COL_TG + gx] - soft_div_rn((double)fluxf[0][c], P.by_dt, dt);
        }
      }
      half_sources(j);   // S_RHOF in FP32: its doubles were read before the last barrier
    }
    __syncthreads();
    half_active();
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int c = threadIdx.x + j * blockDim.x;
      if (c >= ncell) continue;
      const int k = c / COL_TG, gx = c % COL_TG;
      float ff[2] = {0.0f, 0.0f};
      if ((act >> j) & 1u) {
        const float* const sf[2] = {FF(S_RHOF) + gx, FF(S_RHOF) + ncell + gx};
        flux_integrals<COL_TG, 2>(sf, dgzhf, k, kc[j], restf[j], bmn_h[k], bmx_f[k], ff);
      }
      FF(S_F)[c] = ff[0];
      FF(S_F)[ncell + c] = ff[1];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int c = threadIdx.x + j * blockDim.x;
      const int k = c / COL_TG, g = g0 + c % COL_TG;
      if (c >= ncell || g >= G || k < kmin + 1 || k > kmax) continue;
      const float* f0 = FF(S_F);
      const float* f1 = f0 + ncell;
      FF(S_DKINV)[c] = FF(S_DKINV)[c] - (f0[c] - f0[c - COL_TG]) * rdgzhf[k];
      FF(S_DRHOGW)[c] = FF(S_DRHOGW)[c] - (f1[c] - f1[c - COL_TG]) * rdgzhf[k];
    }
  }
  __syncthreads();

  // ---- apply the tendencies (mod_precip_transport.cpp:956-989); a zero
  //      tendency leaves its field as it is
#pragma unroll 1
  for (int c = threadIdx.x; c < ncell; c += blockDim.x, odd >>= 1) {
    const int k = c / COL_TG, gx = c % COL_TG, g = g0 + gx;
    if (g >= G) continue;
    const bool full = odd & 1u;   // a zero tendency times an infinity or a NaN is none
    const size_t i = off + (size_t)k * G + g;
    const size_t ic = (size_t)l * G + g;
    const size_t iq = offq + (size_t)k * G + g;
    double rhoge = P.rhoge[i], rhog = P.rhog[i], rw = P.rhogw[i];
    double rvx = P.rhogvx[i], rvy = P.rhogvy[i], rvz = P.rhogvz[i];
    const double zz = P.z[i];
    const double rqr = P.rhogq[iq + (size_t)I_QR * KG], rqs = P.rhogq[iq + (size_t)I_QS * KG],
                 rqg = P.rhogq[iq + (size_t)I_QG * KG], rqi = OPT ? P.rhogq[iq + (size_t)I_QI * KG] : 0.0;
    loaded(rhoge), loaded(rhog), loaded(rw), loaded(rvx), loaded(rvy), loaded(rvz), loaded(zz);
    loaded(rqr), loaded(rqs), loaded(rqg);
    if (OPT) loaded(rqi);
    const double de = F(S_DRHOE)[c], dphi = F(S_DRHOPHI)[c];
    if (!fp_is_zero(de)) rhoge = rhoge + de;
    if (!fp_is_zero(dphi)) rhoge = rhoge + dphi;
    if (MIX) {
      FF(S_KINH)[c] = FF(S_KINH)[c] + FF(S_DKINH)[c];
      FF(S_KINV)[c] = FF(S_KINV)[c] + FF(S_DKINV)[c];
    } else {
      if (!fp_is_zero(F(S_DKINH)[c])) F(S_KINH)[c] = F(S_KINH)[c] + F(S_DKINH)[c];
      if (!fp_is_zero(F(S_DKINV)[c])) F(S_KINV)[c] = F(S_KINV)[c] + F(S_DKINV)[c];
    }
    if (MIX) {
      // the FP32 momentum tendencies along the FP32 unit vectors, added to the FP64 state
      const float du = FF(S_DRHOGU)[c], dv = FF(S_DRHOGV)[c];
      if (du != 0.0f || dv != 0.0f || full) {
        P.rhogvx[i] = rvx = rvx + soft_f2d(__fmaf_rn(dv, uvf[3 * COL_TG + gx], __fmul_rn(du, uvf[gx])));
        P.rhogvy[i] = rvy = rvy + soft_f2d(__fmaf_rn(dv, uvf[4 * COL_TG + gx], __fmul_rn(du, uvf[1 * COL_TG + gx])));
        P.rhogvz[i] = rvz = rvz + soft_f2d(__fmaf_rn(dv, uvf[5 * COL_TG + gx], __fmul_rn(du, uvf[2 * COL_TG + gx])));
      }
    } else {
      const double du = F(S_DRHOGU)[c], dv = F(S_DRHOGV)[c];
      if (!(fp_is_zero(du) && fp_is_zero(dv)) || full) {
        P.rhogvx[i] = rvx = rvx + du * P.ix[ic] + dv * P.jx[ic];
        P.rhogvy[i] = rvy = rvy + du * P.iy[ic] + dv * P.jy[ic];
        P.rhogvz[i] = rvz = rvz + du * P.iz[ic] + dv * P.jz[ic];
      }
    }
    const double dw = MIX ? soft_f2d(FF(S_DRHOGW)[c]) : F(S_DRHOGW)[c];
    if (!fp_is_zero(dw)) {
      rw = rw + dw;
      P.rhogw[i] = rw;
    }
    if (!MIX) F(S_DRHOGW)[c] = rw;   // MIX: the FP32 view of this slot is still being read
    // tracers in order QV..QG (QV, QC and QI add exact zeros; the -0 that makes a +0 is left to final_cell)
    auto add = [&](int n, double rq, double dq) {
      if (fp_is_zero(dq) && !full) return;
      soft_branch();
      P.rhogq[iq + (size_t)n * KG] = rq + dq;
      rhog = rhog + dq;
      rhoge = rhoge - dq * GRAV * zz;
    };
    add(I_QR, rqr, F(S_DQR)[c]);
    if (OPT && ntr == 4) add(I_QI, rqi, F(S_DQI)[c]);
    add(I_QS, rqs, F(S_DQS)[c]);
    add(I_QG, rqg, F(S_DQG)[c]);
    P.rhog[i] = rhog;
    F(S_RHOF)[c] = rhog;
    F(S_DQR)[c] = rhoge;   // for the final pass
    // (the horizontal kinetic energy of the updated state times rhog)
    if (!MIX && !kin2kin && k >= kmin && k <= kmax) F(S_DKINH)[c] = 0.5 * (rvx * rvx + rvy * rvy + rvz * rvz);
    if (MIX) {
      const float rhogf = soft_d2f(rhog);
      FF(S_KINH)[ncell + c] = rhogf;   // rhog after the transport, for the FP32 kinetic energies
      FF(S_DKINV)[c] = soft_d2f(rw);   // and rhogw
      // the horizontal kinetic energy carried by the transport less that of the updated state
      if (!kin2kin && k >= kmin && k <= kmax)
        FF(S_KINH)[c] = FF(S_KINH)[c] - kin_h_f(soft_d2f(rvx), soft_d2f(rvy), soft_d2f(rvz), rhogf);
    }
  }
  __syncthreads();

  // ---- KIN2KIN (mod_precip_transport.cpp:1012-1068), with the switch: the
  //      momentum is rescaled so that the kinetic energy carried by the
  //      transport is kept, horizontal on [kmin, kmax], vertical on
  //      [kmin, kmax+1] (where the carried energy is zero at kmin and kmax+1)
  if (kin2kin) {
#pragma unroll 1
    for (int c = threadIdx.x; c < ncell; c += blockDim.x) {
      const int k = c / COL_TG, gx = c % COL_TG, g = g0 + gx;
      if (g >= G || k < kmin || k > kmax + 1) continue;
      const size_t i = off + (size_t)k * G + g;
      const double rhog = F(S_RHOF)[c];
      if (k <= kmax) {
        const Divisor by_rhog(rhog);
        const double kin_h0 = soft_div(MIX ? (double)FF(S_KINH)[c] : F(S_KINH)[c], by_rhog.s, rhog);
        double vx_t = soft_div(P.rhogvx[i], by_rhog.s, rhog), vy_t = soft_div(P.rhogvy[i], by_rhog.s, rhog),
               vz_t = soft_div(P.rhogvz[i], by_rhog.s, rhog);
        const double kin_h = 0.5 * (vx_t * vx_t + vy_t * vy_t + vz_t * vz_t);
        if (kin_h > 1.0E-20) {
          const double r = sqrtR(fabs(quo(kin_h0, kin_h)));
          vx_t = vx_t * r;
          vy_t = vy_t * r;
          vz_t = vz_t * r;
        }
        P.rhogvx[i] = vx_t * rhog;
        P.rhogvy[i] = vy_t * rhog;
        P.rhogvz[i] = vz_t * rhog;
      }
      const double c2w0 = quo(afact[k], P.gsgam2[i]) * P.gsgam2h[i];
      const double c2w1 = quo(bfact[k], P.gsgam2[i - G]) * P.gsgam2h[i];
      const double rhogh = c2w0 * rhog + c2w1 * F(S_RHOF)[c - COL_TG];
      const double kin_v0 = quo(MIX ? (double)FF(S_KINV)[c] : F(S_KINV)[c], rhogh);
      double w_t = quo(P.rhogw[i], rhogh);
      const double kin_v = 0.5 * (w_t * w_t);
      if (kin_v > 1.0E-20) w_t = w_t * sqrtR(fabs(quo(kin_v0, kin_v)));
      P.rhogw[i] = w_t * rhogh;
    }
  }

  // ---- KIN2EIN (mod_precip_transport.cpp:991-1011): tmp2 and the vertical
  //      kinetic energy of the updated state
  //      (and, in the reference configuration's kernel, the metric factors
  //      W2Cfact of each interior cell for the final pass, in the dead slots
  //      S_DRHOGW / S_DRHOGV, read after rw)
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int c = threadIdx.x + j * blockDim.x;
    if (c >= ncell || kin2kin) continue;
    const int k = c / COL_TG, gx = c % COL_TG, g = g0 + gx;
    if (MIX) {
      // FP32: the change of the vertical kinetic energy of half level k by
      // the transport, (KINV + its tendency) - the energy of the updated
      // state, in the FP32 half of S_DRHOPHI (zero where there is none), and
      // W2Cfact of the interior cells in the two halves of S_DRHOE
      float dkv = 0.0f;
      if (g < G && k >= kmin + 1 && k <= kmax) {
        dkv = FF(S_KINV)[c] - kin_v_f(FF(S_DKINV)[c], r_c2w0f[j], r_c2w1f[j], FF(S_KINH)[ncell + c],
                                      FF(S_KINH)[ncell + c - COL_TG]);
      }
      FF(S_DRHOPHI)[c] = dkv;
      if (g < G && k >= kmin && k <= kmax) {
        const float gsgf = FF(S_VJ)[ncell + c], ghu = FF(S_VI)[ncell + c + COL_TG];
        FF(S_DRHOE)[c] = __fdiv_rn(__fmul_rn(cff[k], gsgf), ghu);
        FF(S_DRHOE)[ncell + c] = __fdiv_rn(__fmul_rn(dff[k], gsgf), ghu);
      }
      continue;
    }
    F(S_DRHOE)[c] = 0.0;
    F(S_DRHOPHI)[c] = 0.0;
    if (g >= G) continue;
    const size_t i = off + (size_t)k * G + g;
    const bool hk = (k >= kmin + 1 && k <= kmax);
    const double rw = hk ? F(S_DRHOGW)[c] : 0.0;
    if (k >= kmin && k <= kmax) {
      const Divisor by_gh(P.gsgam2h[i + G]);
      const double w2c0 = div_rn(cfact[k] * P.gsgam2[i], by_gh);
      const double w2c1 = div_rn(dfact[k] * P.gsgam2[i], by_gh);
      F(S_DRHOE)[c] = F(S_KINH)[c] + (w2c0 * F(S_KINV)[c + COL_TG] + w2c1 * F(S_KINV)[c]);
      if (!OPT) {
        F(S_DRHOGW)[c] = w2c0;
        F(S_DRHOGV)[c] = w2c1;
      }
    }
    if (hk) F(S_DRHOPHI)[c] = quo(0.5 * (rw * rw), r_c2w0[j] * F(S_RHOF)[c] + r_c2w1[j] * F(S_RHOF)[c - COL_TG]);
  }
  __syncthreads();

  // ---- per cell: KIN2EIN, final thermodynamics, saturation adjustment,
  //      negative filter, outputs.  The saturation-adjustment Newton
  //      iteration runs only in saturated cells, a few percent of them; a
  //      tile's would share one warp, which issues one FP64 instruction per
  //      64 cycles where the SM issues one per 19.  So the saturated cells are
  //      left as they are (rhoge after KIN2EIN stored), listed, and finished
  //      by nsw6_satadj_kernel, whose warps are full and fill every SM.
  __shared__ int nqueue;
  __shared__ unsigned qbase;
  if (threadIdx.x == 0) nqueue = 0;
  __syncthreads();
  const float lovr_f = float(C.LovR_liq);
  int* qcell = reinterpret_cast<int*>(F(S_RHOF2));   // the tile's saturated cells (S_RHOF2 is dead by now)
#pragma unroll 1
  for (int c = threadIdx.x; c < ncell; c += blockDim.x) {
    const int k = c / COL_TG, gx = c % COL_TG, g = g0 + gx;
    if (g >= G) continue;
    const size_t i = off + (size_t)k * G + g;
    const bool interior = (k >= kmin && k <= kmax);
    const size_t iq = offq + (size_t)k * G + g;
    double rq[6];
#pragma unroll
    for (int n = 0; n < 6; ++n) loaded(rq[n] = P.rhogq[iq + (size_t)n * KG]);
    const double gsg = P.gsgam2[i];
    loaded(gsg);
    const double rhog = F(S_RHOF)[c];
    const Divisor by_rhog(rhog);   // of the cell's quotients (correctly rounded, as the reference's divisions)
    double rhoge = F(S_DQR)[c];
    if (MIX && interior && !kin2kin) {
      // FP32 kinetic energies: the horizontal energy after the transport
      // against before (with its tendency), the vertical energies' changes
      // weighted by W2Cfact; their sum enters the FP64 internal energy
      const float dke = FF(S_KINH)[c] +
                        __fmaf_rn(FF(S_DRHOE)[c], FF(S_DRHOPHI)[c + COL_TG],
                                  __fmul_rn(FF(S_DRHOE)[ncell + c], FF(S_DRHOPHI)[c]));
      if (dke != 0.0f) rhoge = rhoge + soft_f2d(dke);
    } else if (interior && !kin2kin) {
      const double tmp_h = div_rn(F(S_DKINH)[c], by_rhog);
      double w2c0, w2c1;
      if (!OPT) {
        w2c0 = F(S_DRHOGW)[c];
        w2c1 = F(S_DRHOGV)[c];
      } else {
        const Divisor by_gh(P.gsgam2h[i + G]);
        w2c0 = div_rn(cfact[k] * P.gsgam2[i], by_gh);
        w2c1 = div_rn(dfact[k] * P.gsgam2[i], by_gh);
      }
      const double tmp = tmp_h + (w2c0 * F(S_DRHOPHI)[c + COL_TG] + w2c1 * F(S_DRHOPHI)[c]);
      rhoge = rhoge + (F(S_DRHOE)[c] - tmp);
    }
    if (final_cell<ColumnMath, MIX, OPT>(P, C, mth, ice_adj, lovr_f, i, iq, KG, interior, rhog, by_rhog, rhoge, rq, gsg,
                                         false, k, g, l)) {
      P.rhoge[i] = rhoge;   // its adjustment starts from here
      qcell[atomicAdd(&nqueue, 1)] = c;
    }
    if (k == kmin) {
      const size_t ic = (size_t)l * G + g;
      const size_t r0 = (size_t)l * G + g, r1 = P.prec_ld + r0;
      const double* acc = S.colacc;
      P.precip[r0] = plus_zero(acc[0 * COL_TG + gx]);
      P.precip[r1] = plus_zero(acc[1 * COL_TG + gx]);
      P.iso1[r0] = 0.0;
      P.iso1[r1] = 0.0;
      P.iso2[r0] = 0.0;
      P.iso2[r1] = 0.0;
      P.precip_lh_heat[ic] = plus_zero(acc[2 * COL_TG + gx]);
      P.precip_rhoe[ic] = plus_zero(acc[3 * COL_TG + gx]);
      P.precip_rhophi[ic] = plus_zero(acc[4 * COL_TG + gx]);
      P.precip_rhokin[ic] = plus_zero(acc[5 * COL_TG + gx]);
    }
  }
  __syncthreads();
  // the tile's saturated cells join the list (satq[0] counts them)
  if (threadIdx.x == 0) qbase = nqueue > 0 ? atomicAdd(P.satq, (unsigned)nqueue) : 0u;
  __syncthreads();
  for (int e = threadIdx.x; e < nqueue; e += blockDim.x) {
    const int c = qcell[e];
    P.satq[1 + qbase + e] = (unsigned)(off + (size_t)(c / COL_TG) * G + g0 + c % COL_TG);
  }
}

// ------------------------------------------------------ saturation adjustment
// The saturated cells the column kernel listed (P.satq): the cell's state
// after KIN2EIN is formed again exactly as there, the saturation-adjustment
// Newton iteration runs and the cell is finished (final_cell).  One thread per
// cell, grid-stride over the list, whose length only the device knows.  Bound by
// the latency of the iteration's chain where the list is short, by the FP64 pipe
// where it is long: CTAs of one warp spread a short list over all SMs (with 128
// threads some had twice the warps of others), the tables through L1.  Twelve
// mixed steps of 2500 x 42 1.593 -> 1.561 ms, one region's FP64 step 1.037 ->
// 1.030 ms, ten regions the same.
constexpr int SAT_THREADS = 32;
// CTAs: enough for a sixteenth of the cells in one sweep, so that the last ones
// level out (some 4 percent are saturated in ordinary weather); at least 8 an
// SM, for a small call that is saturated throughout, and no more than 64, whose
// start costs.  Any number of saturated cells is handled, the loop strides over
// the list; where 37 percent are (a state 1.6 times as moist) a region's call
// takes two or three uneven sweeps, 1144 us in FP64 and 667 in mixed precision
// where 64 CTAs an SM take 1123 and 650; ten regions take the same.
inline int sat_blocks(long long cells) {
  const long long n = cells / (16 * SAT_THREADS);
  return (int)(n < 152 * 8 ? 152 * 8 : n > 152 * 64 ? 152 * 64 : n);
}

template <bool MIX, bool OPT>
__global__ void __launch_bounds__(SAT_THREADS) nsw6_satadj_kernel(Problem P, Consts C) {
  const unsigned n = P.satq[0];
  if (blockIdx.x * blockDim.x >= n) return;
  const ColumnMath mth{FastMath(P.fmtab), P.math_lib != 0};
  const int G = P.gall;
  const size_t KG = (size_t)P.kall * G;
  const bool ice_adj = OPT && C.opt_expice == 0.0;
  const float lovr_f = float(C.LovR_liq);
  for (unsigned e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const size_t i = P.satq[1 + e];
    const int l = (int)(i / KG);
    const size_t r = i - (size_t)l * KG;
    const int k = (int)(r / G), g = (int)(r - (size_t)k * G);
    const double rhog = P.rhog[i];
    const size_t iq = (size_t)l * NQ * KG + r;
    const double rhoge = P.rhoge[i], gsg = P.gsgam2[i];
    double rq[6];
#pragma unroll
    for (int n = 0; n < 6; ++n) loaded(rq[n] = P.rhogq[iq + (size_t)n * KG]);
    final_cell<ColumnMath, MIX, OPT>(P, C, mth, ice_adj, lovr_f, i, iq, KG, true, rhog, Divisor(rhog), rhoge, rq, gsg, true,
                                     k, g, l);
  }
}

// ------------------------------------------------------------------ launchers
// Columns of a CTA and cells of a thread.  16 columns (8 above 64 levels, for
// shared memory: two CTAs an SM); a call of fewer columns than that fills the
// SMs with gets 8 or 4, which spread it over more SMs with fewer cells a
// thread.
struct ColumnShape {
  int tg, threads, nj;
};
inline ColumnShape column_shape(int K, int gall, int lall) {
  ColumnShape s;
  s.tg = K <= 64 ? 16 : 8;
  auto ctas = [&](int tg) { return (long long)((gall + tg - 1) / tg) * lall; };
  if (s.tg == 16 && ctas(16) <= 2 * 152 && K * 8 <= COL_THREADS_MAX) s.tg = 8;
  if (ctas(8) <= 152 && K * 4 <= COL_THREADS_MAX) s.tg = 4;
  const int ncell = K * s.tg;
  s.nj = (ncell + COL_THREADS_MAX - 1) / COL_THREADS_MAX;
  s.threads = ((ncell + s.nj - 1) / s.nj + 31) / 32 * 32;
  return s;
}

inline size_t column_smem_bytes(int K, int tg, bool opt) {
  const size_t nslot = opt ? S_COUNT_OPT : S_COUNT;
  const size_t nrow = opt ? 8 : 6;
  return sizeof(double) * (nslot * K * tg + GF_COUNT * K + 6 * tg + 2 * K) + sizeof(int) * 2 * nrow * K +
         sizeof(float) * (8 * K + 6 * tg);
}

// Calls f(kernel) for the instantiation of a shape; false: there is none.
template <bool MIX, bool OPT, class Fn>
bool with_column_kernel(int tg, int nj, Fn f) {
  if (tg == 16 && nj == 1) f(nsw6_column_kernel<16, 1, MIX, OPT>);
  else if (tg == 16 && nj == 2) f(nsw6_column_kernel<16, 2, MIX, OPT>);
  else if (tg == 16 && nj == 3) f(nsw6_column_kernel<16, 3, MIX, OPT>);
  else if (tg == 8 && nj == 1) f(nsw6_column_kernel<8, 1, MIX, OPT>);
  else if (tg == 8 && nj == 2) f(nsw6_column_kernel<8, 2, MIX, OPT>);
  else if (tg == 8 && nj <= 4) f(nsw6_column_kernel<8, 4, MIX, OPT>);
  else if (tg == 4 && nj == 1) f(nsw6_column_kernel<4, 1, MIX, OPT>);
  else return false;
  return true;
}

// Raises a kernel's dynamic shared-memory limit to what the device allows a
// block beside the kernel's own static shared memory.
template <class Kernel>
cudaError_t raise_smem_limit(Kernel k, int optin) {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, k);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)a.sharedSizeBytes);
}

template <bool MIX, bool OPT>
cudaError_t prepare_column(int optin) {
  cudaError_t e = cudaSuccess;
  const int shapes[7][2] = {{16, 1}, {16, 2}, {16, 3}, {8, 1}, {8, 2}, {8, 4}, {4, 1}};
  for (const auto& s : shapes)
    with_column_kernel<MIX, OPT>(s[0], s[1], [&](auto k) {
      const cudaError_t r = raise_smem_limit(k, optin);
      if (r != cudaSuccess) e = r;
    });
  return e;
}

// The column kernel and the saturation adjustment.
template <bool MIX, bool OPT>
cudaError_t run_column(const Problem& P, const Consts& C, cudaStream_t stream) {
  const ColumnShape s = column_shape(P.kall, P.gall, P.lall);
  const dim3 grid((P.gall + s.tg - 1) / s.tg, P.lall);
  const size_t sm = column_smem_bytes(P.kall, s.tg, OPT);
  if (!with_column_kernel<MIX, OPT>(s.tg, s.nj, [&](auto k) { k<<<grid, s.threads, sm, stream>>>(P, C); }))
    return cudaErrorInvalidConfiguration;
  nsw6_satadj_kernel<MIX, OPT><<<sat_blocks((long long)P.lall * P.kall * P.gall), SAT_THREADS, 0, stream>>>(P, C);
  return cudaGetLastError();
}

}  // namespace nsw6
