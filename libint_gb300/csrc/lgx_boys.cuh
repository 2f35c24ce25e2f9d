// Boys function evaluators of the register kernels (F_0..F_MMAX at compile-
// time MMAX, times the primitive prefactor), FP64 and FP32.  The program
// kernels' runtime-mmax evaluators are boys_to_stage (lgx_warp.cuh).
#pragma once
#include "lgx_kernels.cuh"

namespace lgx {

// The store kernels' FP64 evaluation for values that are rounded to FP32 next,
// once the branch and the grid point are chosen (rk_boys_b64): the 1/64 grid's
// pre-divided table, k the grid point and md = T_k - T, every m directly when
// MMAX <= 2, else the top m and the downward recursion with e^{-T} as the
// tabulated e^{-T_k} times the series of e^{md}; 4 terms, 1.6e-10 of F_m, whose
// half-ulp is 6e-8.  asym: sqrt(pi/T)/2 and the upward recursion without the
// e^{-T} terms, 1/sqrt(T) by one FP64 Newton step from the FP32 estimate.
template <int MMAX>
__device__ __forceinline__ void rk_boys_core(const double* __restrict__ tay, double T, bool asym,
                                             int k, double md, double* F) {
  static_assert(MMAX <= 6, "asymptotic branch without e^{-T} is exact to 2e-15 only for m <= 6");
  if (asym) {
    const double r0 = f2d_int(rsqrtf(d2f_int(T)));  // relative error <= ~3e-7
    const double rs = fma(0.5 * r0, fma(-(T * r0), r0, 1.0), r0);
    const double oo2T = 0.5 * (rs * rs);
    double f = 0.88622692545275801365 * rs;
    F[0] = f;
#pragma unroll
    for (int m = 0; m < MMAX; ++m) {
      f *= (2 * m + 1) * oo2T;
      F[m + 1] = f;
    }
    return;
  }
  const double* row = tay + (k * (kBoysMaxM + 1)) * kBoysTaylorStride;
  auto series = [&](const double* c) {
    double s = __ldg(c + 3);
    s = fma(s, md, __ldg(c + 2));
    s = fma(s, md, __ldg(c + 1));
    return fma(s, md, __ldg(c));
  };
  if (MMAX <= 2) {
#pragma unroll
    for (int m = 0; m <= MMAX; ++m) F[m] = series(row + m * kBoysTaylorStride);
  } else {
    double s = series(row + MMAX * kBoysTaylorStride);
    F[MMAX] = s;
    double e = 1.0 / 6.0;
    e = fma(e, md, 0.5);
    e = fma(e, md, 1.0);
    e = fma(e, md, 1.0);
    const double eT = __ldg(row + 7) * e;
    const double twoT = 2.0 * T;
#pragma unroll
    for (int m = MMAX - 1; m >= 0; --m) {
      s = fma(twoT, s, eT) * (1.0 / (2 * m + 1));
      F[m] = s;
    }
  }
}

// The register kernels' FP64 Boys function, F_m(T) pfac, from the fine tables.
//  T <= 50: c0 + md (c1 + md (c2 + md (c3 + c4 md))), md = T_j - T, the inner
//   bracket in FP32; every m directly for MMAX <= 2, else the top m, and
//   e^{-T} = e^{-T_j} e^{md} by the same kind of series
//   (MMAX > 2: the downward recursion from there).
//  T > 50: sqrt(pi/T)/2 and the upward recursion without its e^{-T} terms (below
//   1.7e-15 of F_6 there).  Not the top m and the downward recursion that the
//   lanes below 50 run: that gives F_0 the error of F_MMAX, 2.3e-15 instead of
//   2.4e-16 at MMAX = 6, and zero where F_MMAX underflows.
// What bounds it: the FP64 pipe (2 lanes per cycle and SM), so everything that
// only chooses (branch, grid point) or lies below 2^-32 runs in integer and
// FP32 instructions: per m 3 FP64 operations instead of 5 on the 1/64 grid, and
// 1 instead of 4 for the grid point.  The tables (0.8 MB for MMAX = 0, 2.5 MB
// for 2) stay in L2.
// Error against 128-bit values, root mean square over T <= 50, this and the
// six-term FP64 series on the 1/64 grid: F_0 6.3e-17 and 6.3e-17 (MMAX = 0),
// 1.63e-16 and 1.67e-16 (MMAX = 6), F_6 6.6e-17 and 6.7e-17; beyond 50 the same.
template <int MMAX>
__device__ __forceinline__ void rk_boys(const double* __restrict__ fine, double T, double pfac,
                                        double* F) {
  static_assert(MMAX <= kBoysFineM, "fine tables and the asymptotic branch end at m = 6");
  const float Tf = d2f_int(T);
  const bool asym = Tf > float(kBoysTmax);
  if (asym) {
    const double rs = rsqrt(T);
    const double oo2T = 0.5 * (rs * rs);
    double f = (0.88622692545275801365 * pfac) * rs;
    F[0] = f;
#pragma unroll
    for (int m = 0; m < MMAX; ++m) {
      f *= (2 * m + 1) * oo2T;
      F[m + 1] = f;
    }
    return;
  }
  const int j = __float2int_rn(Tf * float(kBoysFineInv));
  const double md = fma(i2d_int(j), 1.0 / kBoysFineInv, -T);
  const float mdf = d2f_int(md);
  const double2* row = reinterpret_cast<const double2*>(fine + boys_fine_off(MMAX) +
                                                        j * boys_fine_cols(MMAX));
  auto series = [&](int e) {  // of the row's entry e
    const double2 a = __ldg(row + 2 * e), b = __ldg(row + 2 * e + 1);
    const float c3 = __int_as_float(__double2loint(b.y)), c4 = __int_as_float(__double2hiint(b.y));
    double s = fma(md, f2d_int(fmaf(mdf, c4, c3)), b.x);
    s = fma(md, s, a.y);
    return fma(md, s, a.x);
  };
  if (MMAX <= 2) {
#pragma unroll
    for (int m = 0; m <= MMAX; ++m) F[m] = series(m) * pfac;
    return;
  }
  double s = series(0) * pfac;
  // e^{md} = 1 + md (1 + md (1/2 + md (1/6 + md/24)))
  double e = fma(md, f2d_int(fmaf(mdf, 1.0f / 24.0f, 1.0f / 6.0f)), 0.5);
  e = fma(md, e, 1.0);
  e = fma(md, e, 1.0);
  const double eTp = (__ldg(row + 2).x * pfac) * e;
  F[MMAX] = s;
  const double twoT = 2.0 * T;
#pragma unroll
  for (int m = MMAX - 1; m >= 0; --m) {
    s = fma(twoT, s, eTp) * (1.0 / (2 * m + 1));
    F[m] = s;
  }
}

// The FP64 Boys step of the attenuated operators (register kernels of the J/K
// passes): F = the core integrals times pfac, with s = omega^2 / (omega^2 + rho)
// (libint's erf_coulomb_gm_eval / erfc_coulomb_gm_eval,
// include/libint2/boys.h:1913-1980)
//   erf(omega r)/r  (op 1):  s^{m+1/2} F_m(s T)
//   erfc(omega r)/r (op 2):  F_m(T) - s^{m+1/2} F_m(s T)
// (s T <= T, so the same grid serves).  s is a division and sqrt(s) a square
// root: both from one reciprocal square root of omega^2 + rho would double the
// error of s^{m+1/2} (at m = 4 1.4e-15 instead of 8e-16 of F_m).  erf needs no
// F_m(T).  Returns false when the integrals vanish: erf at omega = 0, and erfc
// where s T > 50, as both parts are then asymptotic and equal (their difference
// is below e^-50 of F_m; evaluated, it is the rounding noise of two equal sums).
template <int MMAX>
__device__ __forceinline__ bool rk_boys_att(const double* __restrict__ fine, int op, double omega2,
                                            double T, double rho, double pfac, double* F) {
  if (!(omega2 > 0.0)) {
    if (op == 1) return false;
    rk_boys<MMAX>(fine, T, pfac, F);
    return true;
  }
  const double s = omega2 / (omega2 + rho);
  const double sT = s * T;
  if (op == 2 && d2f_int(sT) > float(kBoysTmax)) return false;
  double G[MMAX + 1];
  rk_boys<MMAX>(fine, sT, pfac * sqrt(s), G);
  if (op == 1) {
    double f = 1.0;
#pragma unroll
    for (int m = 0; m <= MMAX; ++m, f *= s) F[m] = m == 0 ? G[0] : f * G[m];
    return true;
  }
  rk_boys<MMAX>(fine, T, pfac, F);
  double f = s;
  F[0] -= G[0];
#pragma unroll
  for (int m = 1; m <= MMAX; ++m, f *= s) F[m] = fma(-f, G[m], F[m]);
  return true;
}

// The mixed scheme's FP64 Boys function of an FP32 quartet (store kernels), given its
// argument T = T.hi + T.lo in double-float (ds_boys_arg): the branch and the
// grid point come from T.hi; the offset md = T_k - T = (T_k - T.hi) - T.lo,
// where T_k - T.hi is exact in FP32 (T_k = k/64 and T.hi are within a
// factor 2 of each other for k >= 1, Sterbenz; 0 - T.hi for k = 0), both
// parts converted to FP64 with integer operations and subtracted in FP64;
// T itself in FP64 (one addition) for the asymptotic branch and the
// recursion.  T.hi <= 50 gives k <= 3200 < kBoysRows, and near T = 50 either
// branch is exact (the asymptotic one drops Q(m+1/2, T) < 2e-15).  The
// values are rounded to FP32 next, so the series stop at 4 terms: relative
// error below 1.6e-10 (|md| <= 1/128), 400 times under the FP32 half-ulp.
template <int MMAX>
__device__ __forceinline__ void rk_boys_b64(const double* __restrict__ tay, dsf T, double* F) {
  const bool asym = T.hi > float(kBoysTmax);
  const int k = asym ? 0 : __float2int_rn(T.hi * float(kBoysInvDT));
  const float mdh = __fadd_rn(__fmul_rn(float(k), float(kBoysDT)), -T.hi);
  const double md = f2d_int(mdh) - f2d_int(T.lo);
  if (MMAX <= 2 && !asym) {  // direct Taylor series: T itself is not needed
    rk_boys_core<MMAX>(tay, 0.0, false, k, md, F);
    return;
  }
  const double T64 = f2d_int(T.hi) + f2d_int(T.lo);
  rk_boys_core<MMAX>(tay, T64, asym, k, md, F);
}

// The Boys function of the mixed scheme's J/K kernels times the FP32
// prefactor, F_m(T) pfac for T = T.hi + T.lo in double-float (ds_boys_arg),
// with no FP64 instruction: every value is a leading FP32 part plus an FP32
// correction, rounded once in the product by pfac.
//  T <= 50: F_m(T) = hi_m + [lo_m + md F_{m+1} + md^2/2 (F_{m+2} + md/3
//   (F_{m+3} + md/4 F_{m+4}))] of the split table, for every m directly; md = T_k - T =
//   (T_k - T.hi) - T.lo, whose first difference is exact (Sterbenz) and whose
//   two parts multiply F_{m+1} one by one: with |md| <= 1/128 the bracket is
//   right to 2^-31 of F_m, 1/128 of the FP32 half-ulp; the series stops at
//   2.5e-13.
//  T > 50: r = T^{-1/2} and u = 1/(2T) as hi + lo (boys_asym), F_0 =
//   sqrt(pi)/2 r, F_{m+1} = (2m+1) u F_m without the e^{-T} terms.
// Error against 128-bit values, this and rk_boys_b64 (pfac = 1): 5.92e-8 at most
// and 2.5e-8 root mean square for both, every m <= 6, T up to 300 (the FP32
// rounding); the product by pfac is the same rounding here, a second one there.
// The store kernels keep rk_boys_b64: they hand out the integrals one by one,
// and this evaluation, although as close to the exact values, rounds about
// one F_m in a thousand (and every product by pfac) the other way.
// What bounds it: the gathers (2 LDG.128 for m <= 1, 5 for m = 6) and FP32
// issue, about 7 instructions per m; evaluated on the FP64 pipe (2 lanes per
// cycle and SM) the same values made that pipe the bound of these kernels
// ((H2O)32 cc-pVDZ mixed pass 218 ms, with this 163 ms).
template <int MMAX>
__device__ __forceinline__ void rk_boys_split(const float* __restrict__ tab, dsf T, float pfac,
                                              float* F) {
  static_assert(MMAX <= kBoysSplitM, "packed split tables end at kBoysSplitM");
  if (T.hi > float(kBoysTmax)) {
    const BoysAsym b = boys_asym(T);
    dsf f = boys_asym_first(b.r);
#pragma unroll
    for (int m = 0; m <= MMAX; ++m) {
      F[m] = boys_asym_out(f, pfac);
      if (m < MMAX) f = boys_asym_step(f, b.u, float(2 * m + 1));
    }
    return;
  }
  constexpr int kCols = boys_split_cols(MMAX);
  const int k = __float2int_rn(T.hi * float(kBoysInvDT));
  const float dh = __fadd_rn(__fmul_rn(float(k), float(kBoysDT)), -T.hi);
  const float md = __fadd_rn(dh, -T.lo);
  const float4* row = reinterpret_cast<const float4*>(tab + boys_split_off(MMAX) + k * kCols);
  float w[kCols];
#pragma unroll
  for (int i = 0; i < kCols / 4; ++i) {
    const float4 v = __ldg(row + i);
    w[4 * i] = v.x;
    w[4 * i + 1] = v.y;
    w[4 * i + 2] = v.z;
    w[4 * i + 3] = v.w;
  }
  const float m2 = 0.5f * md * md, m3 = md * (1.0f / 3.0f), m4 = 0.25f * md;
#pragma unroll
  for (int m = 0; m <= MMAX; ++m) {
    float c = fmaf(m2, fmaf(m3, fmaf(m4, w[m + 4], w[m + 3]), w[m + 2]), w[MMAX + 5 + m]);
    c = fmaf(dh, w[m + 1], fmaf(-T.lo, w[m + 1], c));
    F[m] = fmaf(w[m], pfac, c * pfac);
  }
}

template <int MMAX>
__device__ __forceinline__ void rk_boys(const float* __restrict__ tab, float T, float pfac,
                                        float* F) {
  if (T > float(kBoysTmax)) {
    const float rs = rsqrtf(T);
    const float oo2T = 0.5f * (rs * rs);
    float f = (0.886226925f * pfac) * rs;
    F[0] = f;
#pragma unroll
    for (int m = 0; m < MMAX; ++m) {
      f *= (2 * m + 1) * oo2T;  // e^{-T} < 2e-22 is below FP32 resolution
      F[m + 1] = f;
    }
    return;
  }
  const int k = __float2int_rn(T * float(kBoysInvDT));
  const float d = T - k * float(kBoysDT);
  const float* row = tab + k * kBoysCols;
  const float c3 = -d * (1.0f / 3.0f), c2 = -d * 0.5f, c1 = -d;
  float s = __ldg(row + MMAX + 3);
  s = fmaf(s, c3, __ldg(row + MMAX + 2));
  s = fmaf(s, c2, __ldg(row + MMAX + 1));
  s = fmaf(s, c1, __ldg(row + MMAX));
  s *= pfac;
  F[MMAX] = s;
  if (MMAX > 0) {
    const float eTp = __expf(-T) * pfac;
    const float twoT = 2.0f * T;
#pragma unroll
    for (int m = MMAX - 1; m >= 0; --m) {
      s = fmaf(twoT, s, eTp) * (1.0f / (2 * m + 1));
      F[m] = s;
    }
  }
}

}  // namespace lgx
