// The device Boys evaluators as a batch call (lgx_boys): each thread
// evaluates F_0..F_mmax(T) of one argument with exactly the function a class
// kernel uses, so that the evaluators can be checked on their own.
#include "lgx_boys.cuh"
#include "lgx_warp.cuh"

namespace lgx {
namespace {

// T as a double-float pair.
__device__ __forceinline__ dsf boys_dsf(double T) {
  dsf r;
  r.hi = float(T);
  r.lo = float(T - double(r.hi));
  return r;
}

template <int MMAX>
__device__ void rk_boys_to(const BoysTables& t, int variant, double T, double* out) {
  if (variant == 1) {
    rk_boys<MMAX>(t.fine, T, 1.0, out);
  } else if (variant == 5) {  // the store kernels' FP64 evaluator, rounded as they do
    double f[MMAX + 1];
    rk_boys_b64<MMAX>(t.tay, boys_dsf(T), f);
#pragma unroll
    for (int m = 0; m <= MMAX; ++m) out[m] = double(d2f_int(f[m]));
  } else {
    float f[MMAX + 1];
    if (variant == 8)
      rk_boys_split<MMAX>(t.split, boys_dsf(T), 1.0f, f);
    else
      rk_boys<MMAX>(t.tab32, float(T), 1.0f, f);
#pragma unroll
    for (int m = 0; m <= MMAX; ++m) out[m] = double(f[m]);
  }
}

// Variants 6 and 9: the whole Boys path of the mixed scheme's register kernels
// from primitive-pair data: the double-float records of (Pb, zeta) and (Pk,
// eta), the FP32 prologue's rho and 1/(zeta + eta), then the store kernels'
// argument (ds_boys_arg) and FP64 evaluator rounded to FP32 (6), or the J/K
// kernels' argument (ds_boys_arg_jk) and split tables (9).
template <int MMAX>
__device__ void rk_boys_pairs(const BoysTables& t, int variant, const double* pz, double* out) {
  const PrimPairJKds b = make_jkds(pz[0], pz[1], pz[2], pz[3]);
  const PrimPairJKds k = make_jkds(pz[4], pz[5], pz[6], pz[7]);
  const float zeta = b.hi.w, eta = k.hi.w;
  const float rs = rsqrtf(zeta + eta);
  const float oogpq = rs * rs;
  const float rho = zeta * eta * oogpq;
  if (variant == 9) {
    float f[MMAX + 1];
    rk_boys_split<MMAX>(t.split, ds_boys_arg_jk(b.hi, b.lo, k.hi, k.lo, rho, oogpq), 1.0f, f);
#pragma unroll
    for (int m = 0; m <= MMAX; ++m) out[m] = double(f[m]);
    return;
  }
  double f[MMAX + 1];
  rk_boys_b64<MMAX>(t.tay, ds_boys_arg(b.hi, b.lo, k.hi, k.lo, rho, oogpq), f);
#pragma unroll
  for (int m = 0; m <= MMAX; ++m) out[m] = double(d2f_int(f[m]));
}

// Variant 10: the register J/K kernels' FP64 step of the attenuated operators
// for one (T, rho); zero where it reports that the integrals vanish.
template <int MMAX>
__device__ void rk_boys_att_to(const BoysTables& t, const double* arg, double* out) {
  if (!rk_boys_att<MMAX>(t.fine, t.op, t.omega2, arg[0], arg[1], 1.0, out))
    for (int m = 0; m <= MMAX; ++m) out[m] = 0.0;
}

// Fine tables from the 1/64 grid (hi + lo: the grid values beyond FP64): F_m at
// fine point j by ten terms of its Taylor series about the nearest coarse point
// (distance at most 4/512), the sum rounded once.
__global__ void boys_fine_kernel(const double* hi, const double* lo, double* fine) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= kBoysFineRows) return;
  constexpr int kStep = kBoysFineInv / 64;
  const int k = min((j + kStep / 2) / kStep, kBoysRows - 1);
  const double d = double(k * kStep - j) / kBoysFineInv;  // T_k - T_j
  double F[kBoysFineM + 5];
#pragma unroll
  for (int m = 0; m < kBoysFineM + 5; ++m) {
    const double* c = hi + size_t(k) * kBoysCols + m;
    double s = c[9] / 9.0;
#pragma unroll
    for (int i = 8; i >= 1; --i) s = fma(s, d, c[i]) / i;
    F[m] = c[0] + fma(s, d, lo[size_t(k) * kBoysCols + m]);
  }
#pragma unroll
  for (int M = 0; M <= kBoysFineM; ++M) {
    double* row = fine + boys_fine_off(M) + size_t(j) * boys_fine_cols(M);
    for (int m = M <= 2 ? 0 : M; m <= M; ++m, row += 4) {
      row[0] = F[m];
      row[1] = F[m + 1];
      row[2] = 0.5 * F[m + 2];
      row[3] = __hiloint2double(__float_as_int(float(F[m + 4] / 24.0)),
                                __float_as_int(float(F[m + 3] / 6.0)));
    }
    if (M > 2) {
      row[0] = exp(-double(j) / kBoysFineInv);
      row[1] = 0.0;
    }
  }
}

__global__ void boys_eval_kernel(BoysTables t, int variant, const double* Targ, long long n,
                                 int mmax, double* F) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double out[kBoysMaxM + 1];
  if (variant == 6 || variant == 9) {
    const double* pz = Targ + 8 * i;
    switch (mmax) {
      case 0: rk_boys_pairs<0>(t, variant, pz, out); break;
      case 1: rk_boys_pairs<1>(t, variant, pz, out); break;
      case 2: rk_boys_pairs<2>(t, variant, pz, out); break;
      case 3: rk_boys_pairs<3>(t, variant, pz, out); break;
      case 4: rk_boys_pairs<4>(t, variant, pz, out); break;
      case 5: rk_boys_pairs<5>(t, variant, pz, out); break;
      default: rk_boys_pairs<6>(t, variant, pz, out); break;
    }
    for (int m = 0; m <= mmax; ++m) F[i * (mmax + 1) + m] = out[m];
    return;
  }
  if (variant == 10) {
    const double* arg = Targ + 2 * i;
    switch (mmax) {
      case 0: rk_boys_att_to<0>(t, arg, out); break;
      case 1: rk_boys_att_to<1>(t, arg, out); break;
      case 2: rk_boys_att_to<2>(t, arg, out); break;
      case 3: rk_boys_att_to<3>(t, arg, out); break;
      case 4: rk_boys_att_to<4>(t, arg, out); break;
      case 5: rk_boys_att_to<5>(t, arg, out); break;
      default: rk_boys_att_to<6>(t, arg, out); break;
    }
    for (int m = 0; m <= mmax; ++m) F[i * (mmax + 1) + m] = out[m];
    return;
  }
  const double T = Targ[i];
  if (variant == 0) {
    boys_to_stage(t.tab, t.inv_odd, T, mmax, 1.0, out);
  } else if (variant == 2 || variant == 4 || variant == 7) {  // program kernels, FP32 values
    float f[kBoysMaxM + 1];
    if (variant == 2)
      boys_to_stage(t.tab32, float(T), mmax, 1.0f, f);
    else if (variant == 4)
      boys_b64_stage(t.tay, t.inv_odd, boys_dsf(T), mmax, 1.0f, f);
    else
      boys_split_stage(t.split, boys_dsf(T), mmax, 1.0f, f);
    for (int m = 0; m <= mmax; ++m) out[m] = double(f[m]);
  } else {
    switch (mmax) {
      case 0: rk_boys_to<0>(t, variant, T, out); break;
      case 1: rk_boys_to<1>(t, variant, T, out); break;
      case 2: rk_boys_to<2>(t, variant, T, out); break;
      case 3: rk_boys_to<3>(t, variant, T, out); break;
      case 4: rk_boys_to<4>(t, variant, T, out); break;
      case 5: rk_boys_to<5>(t, variant, T, out); break;
      default: rk_boys_to<6>(t, variant, T, out); break;
    }
  }
  for (int m = 0; m <= mmax; ++m) F[i * (mmax + 1) + m] = out[m];
}

}  // namespace

cudaError_t launch_boys_fine(const double* hi, const double* lo, double* fine, cudaStream_t st) {
  const int block = 128;
  boys_fine_kernel<<<(kBoysFineRows + block - 1) / block, block, 0, st>>>(hi, lo, fine);
  return cudaGetLastError();
}

// variant: as lgx_boys (include/lgx.h), whose checks of the ranges come first.
cudaError_t launch_boys_eval(const BoysTables& t, int variant, const double* T, long long n,
                             int mmax, double* F, cudaStream_t st) {
  const int block = 128;
  const long long grid = (n + block - 1) / block;
  boys_eval_kernel<<<(unsigned)grid, block, 0, st>>>(t, variant, T, n, mmax, F);
  return cudaGetLastError();
}

}  // namespace lgx
