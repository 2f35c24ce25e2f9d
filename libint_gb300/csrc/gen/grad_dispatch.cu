// GENERATED by libint_gb300/codegen/gen_grad.py -- do not edit.
// Run-time dispatch of the register-resident derivative kernels.
#include "../lgx_kernels.cuh"

namespace lgx {
cudaError_t rk_deriv_launch_0000(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_deriv_launch_0010(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_deriv_launch_0011(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_deriv_launch_0020(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_deriv_launch_0021(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_deriv_launch_0030(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_deriv_launch_1010(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_deriv_launch_1011(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_deriv_launch_1020(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_0000(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_0010(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_0011(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_0020(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_0021(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_0022(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_0030(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_0031(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_0032(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_1010(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_1011(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_1020(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_1021(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_1022(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_1030(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_1031(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_1111(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_1120(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_1121(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_1130(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_2011(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_2020(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_2021(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_grad_launch_2030(const EriArgs& a, long long work, int nsm, cudaStream_t st);
cudaError_t rk_one0_launch_0000(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one0_launch_0010(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one0_launch_0011(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one0_launch_0020(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one0_launch_0021(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one0_launch_0022(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one0_launch_0030(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one0_launch_0031(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one0_launch_1010(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one0_launch_1011(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one0_launch_1020(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one0_launch_1021(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one0_launch_1030(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one0_launch_1111(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one0_launch_1120(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one0_launch_2011(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one0_launch_2020(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one1_launch_0000(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one1_launch_0010(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one1_launch_0011(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one1_launch_0020(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one1_launch_0021(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one1_launch_0030(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one1_launch_1010(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one1_launch_1011(const EriArgs& a, int blocks, cudaStream_t st);
cudaError_t rk_one1_launch_1020(const EriArgs& a, int blocks, cudaStream_t st);

cudaError_t rk_grad_launch(int la, int lb, int lc, int ld, const EriArgs& a, long long work, int nsm,
                           cudaStream_t st) {
  switch (((la * 8 + lb) * 8 + lc) * 8 + ld) {
    case 0: return rk_grad_launch_0000(a, work, nsm, st);
    case 8: return rk_grad_launch_0010(a, work, nsm, st);
    case 9: return rk_grad_launch_0011(a, work, nsm, st);
    case 16: return rk_grad_launch_0020(a, work, nsm, st);
    case 17: return rk_grad_launch_0021(a, work, nsm, st);
    case 18: return rk_grad_launch_0022(a, work, nsm, st);
    case 24: return rk_grad_launch_0030(a, work, nsm, st);
    case 25: return rk_grad_launch_0031(a, work, nsm, st);
    case 26: return rk_grad_launch_0032(a, work, nsm, st);
    case 520: return rk_grad_launch_1010(a, work, nsm, st);
    case 521: return rk_grad_launch_1011(a, work, nsm, st);
    case 528: return rk_grad_launch_1020(a, work, nsm, st);
    case 529: return rk_grad_launch_1021(a, work, nsm, st);
    case 530: return rk_grad_launch_1022(a, work, nsm, st);
    case 536: return rk_grad_launch_1030(a, work, nsm, st);
    case 537: return rk_grad_launch_1031(a, work, nsm, st);
    case 585: return rk_grad_launch_1111(a, work, nsm, st);
    case 592: return rk_grad_launch_1120(a, work, nsm, st);
    case 593: return rk_grad_launch_1121(a, work, nsm, st);
    case 600: return rk_grad_launch_1130(a, work, nsm, st);
    case 1033: return rk_grad_launch_2011(a, work, nsm, st);
    case 1040: return rk_grad_launch_2020(a, work, nsm, st);
    case 1041: return rk_grad_launch_2021(a, work, nsm, st);
    case 1048: return rk_grad_launch_2030(a, work, nsm, st);
  }
  return cudaErrorNotSupported;
}

bool rk_grad_available(int la, int lb, int lc, int ld) {
  return la <= 3 && lc <= 3 && la + lb + lc + ld <= 5;
}

cudaError_t rk_deriv_launch(int la, int lb, int lc, int ld, const EriArgs& a, long long work, int nsm,
                           cudaStream_t st) {
  switch (((la * 8 + lb) * 8 + lc) * 8 + ld) {
    case 0: return rk_deriv_launch_0000(a, work, nsm, st);
    case 8: return rk_deriv_launch_0010(a, work, nsm, st);
    case 9: return rk_deriv_launch_0011(a, work, nsm, st);
    case 16: return rk_deriv_launch_0020(a, work, nsm, st);
    case 17: return rk_deriv_launch_0021(a, work, nsm, st);
    case 24: return rk_deriv_launch_0030(a, work, nsm, st);
    case 520: return rk_deriv_launch_1010(a, work, nsm, st);
    case 521: return rk_deriv_launch_1011(a, work, nsm, st);
    case 528: return rk_deriv_launch_1020(a, work, nsm, st);
  }
  return cudaErrorNotSupported;
}

bool rk_deriv_available(int la, int lb, int lc, int ld) {
  return la <= 3 && lc <= 3 && la + lb + lc + ld <= 3;
}

// One quartet over several blocks (derivative order 0 or 1).
cudaError_t rk_one_launch(int deriv, int la, int lb, int lc, int ld, const EriArgs& a, int blocks,
                          cudaStream_t st) {
  switch ((((deriv * 8 + la) * 8 + lb) * 8 + lc) * 8 + ld) {
    case 0: return rk_one0_launch_0000(a, blocks, st);
    case 8: return rk_one0_launch_0010(a, blocks, st);
    case 9: return rk_one0_launch_0011(a, blocks, st);
    case 16: return rk_one0_launch_0020(a, blocks, st);
    case 17: return rk_one0_launch_0021(a, blocks, st);
    case 18: return rk_one0_launch_0022(a, blocks, st);
    case 24: return rk_one0_launch_0030(a, blocks, st);
    case 25: return rk_one0_launch_0031(a, blocks, st);
    case 520: return rk_one0_launch_1010(a, blocks, st);
    case 521: return rk_one0_launch_1011(a, blocks, st);
    case 528: return rk_one0_launch_1020(a, blocks, st);
    case 529: return rk_one0_launch_1021(a, blocks, st);
    case 536: return rk_one0_launch_1030(a, blocks, st);
    case 585: return rk_one0_launch_1111(a, blocks, st);
    case 592: return rk_one0_launch_1120(a, blocks, st);
    case 1033: return rk_one0_launch_2011(a, blocks, st);
    case 1040: return rk_one0_launch_2020(a, blocks, st);
    case 4096: return rk_one1_launch_0000(a, blocks, st);
    case 4104: return rk_one1_launch_0010(a, blocks, st);
    case 4105: return rk_one1_launch_0011(a, blocks, st);
    case 4112: return rk_one1_launch_0020(a, blocks, st);
    case 4113: return rk_one1_launch_0021(a, blocks, st);
    case 4120: return rk_one1_launch_0030(a, blocks, st);
    case 4616: return rk_one1_launch_1010(a, blocks, st);
    case 4617: return rk_one1_launch_1011(a, blocks, st);
    case 4624: return rk_one1_launch_1020(a, blocks, st);
  }
  return cudaErrorNotSupported;
}
}  // namespace lgx
