// The exact-fp32 kernels on fp32 storage, and the choice by storage type.
#include "simt.cuh"

namespace b200fa {

extern template cudaError_t simt_fwd<__nv_bfloat16>(const FwdParams&, cudaStream_t);
extern template cudaError_t simt_bwd<__nv_bfloat16>(const BwdParams&, cudaStream_t);
extern template cudaError_t simt_fwd<__half>(const FwdParams&, cudaStream_t);
extern template cudaError_t simt_bwd<__half>(const BwdParams&, cudaStream_t);

cudaError_t launch_fwd_simt(const FwdParams& p, int dtype, cudaStream_t stream, int* launches) {
  cudaError_t e = cudaErrorInvalidValue;
  if (dtype == kF32) e = simt_fwd<float>(p, stream);
  else if (dtype == kBF16) e = simt_fwd<__nv_bfloat16>(p, stream);
  else if (dtype == kF16) e = simt_fwd<__half>(p, stream);
  if (e == cudaSuccess && launches) *launches += 1;
  return e;
}

cudaError_t launch_bwd_simt(const BwdParams& p, int dtype, cudaStream_t stream, int* launches) {
  cudaError_t e = cudaErrorInvalidValue;
  if (dtype == kF32) e = simt_bwd<float>(p, stream);
  else if (dtype == kBF16) e = simt_bwd<__nv_bfloat16>(p, stream);
  else if (dtype == kF16) e = simt_bwd<__half>(p, stream);
  if (e == cudaSuccess && launches) *launches += 3;
  return e;
}

}  // namespace b200fa
