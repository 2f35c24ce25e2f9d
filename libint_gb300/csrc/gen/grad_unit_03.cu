// GENERATED by libint_gb300/codegen/gen_grad.py -- do not edit.
#include "../lgx_rkgrad.cuh"

namespace lgx {
cudaError_t rk_grad_launch_1121(const EriArgs& a, long long work, int nsm, cudaStream_t st) {
  return rk_grad_launch_one<1, 1, 2, 1>(a, work, nsm, st);
}
cudaError_t rk_grad_launch_1111(const EriArgs& a, long long work, int nsm, cudaStream_t st) {
  return rk_grad_launch_one<1, 1, 1, 1>(a, work, nsm, st);
}
cudaError_t rk_one0_launch_1111(const EriArgs& a, int blocks, cudaStream_t st) {
  return rk_one_launch_one<1, 1, 1, 1, 0>(a, blocks, st);
}
cudaError_t rk_deriv_launch_0021(const EriArgs& a, long long work, int nsm, cudaStream_t st) {
  return rk_deriv_launch_one<0, 0, 2, 1>(a, work, nsm, st);
}
cudaError_t rk_one1_launch_0021(const EriArgs& a, int blocks, cudaStream_t st) {
  return rk_one_launch_one<0, 0, 2, 1, 1>(a, blocks, st);
}
cudaError_t rk_deriv_launch_0020(const EriArgs& a, long long work, int nsm, cudaStream_t st) {
  return rk_deriv_launch_one<0, 0, 2, 0>(a, work, nsm, st);
}
cudaError_t rk_grad_launch_0010(const EriArgs& a, long long work, int nsm, cudaStream_t st) {
  return rk_grad_launch_one<0, 0, 1, 0>(a, work, nsm, st);
}
}  // namespace lgx
