// GENERATED by libint_gb300/codegen/gen_grad.py -- do not edit.
#include "../lgx_rkgrad.cuh"

namespace lgx {
cudaError_t rk_grad_launch_2021(const EriArgs& a, long long work, int nsm, cudaStream_t st) {
  return rk_grad_launch_one<2, 0, 2, 1>(a, work, nsm, st);
}
cudaError_t rk_grad_launch_2011(const EriArgs& a, long long work, int nsm, cudaStream_t st) {
  return rk_grad_launch_one<2, 0, 1, 1>(a, work, nsm, st);
}
cudaError_t rk_one0_launch_2011(const EriArgs& a, int blocks, cudaStream_t st) {
  return rk_one_launch_one<2, 0, 1, 1, 0>(a, blocks, st);
}
cudaError_t rk_deriv_launch_1011(const EriArgs& a, long long work, int nsm, cudaStream_t st) {
  return rk_deriv_launch_one<1, 0, 1, 1>(a, work, nsm, st);
}
cudaError_t rk_one1_launch_1011(const EriArgs& a, int blocks, cudaStream_t st) {
  return rk_one_launch_one<1, 0, 1, 1, 1>(a, blocks, st);
}
cudaError_t rk_one0_launch_0011(const EriArgs& a, int blocks, cudaStream_t st) {
  return rk_one_launch_one<0, 0, 1, 1, 0>(a, blocks, st);
}
cudaError_t rk_one0_launch_0010(const EriArgs& a, int blocks, cudaStream_t st) {
  return rk_one_launch_one<0, 0, 1, 0, 0>(a, blocks, st);
}
}  // namespace lgx
