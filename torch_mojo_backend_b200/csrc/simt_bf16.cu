// The exact-fp32 kernels on bf16 storage.
#include "simt.cuh"

namespace b200fa {

template cudaError_t simt_fwd<__nv_bfloat16>(const FwdParams&, cudaStream_t);
template cudaError_t simt_bwd<__nv_bfloat16>(const BwdParams&, cudaStream_t);

}  // namespace b200fa
