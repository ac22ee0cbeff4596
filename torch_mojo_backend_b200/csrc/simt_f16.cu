// The exact-fp32 kernels on fp16 storage.
#include "simt.cuh"

namespace b200fa {

template cudaError_t simt_fwd<__half>(const FwdParams&, cudaStream_t);
template cudaError_t simt_bwd<__half>(const BwdParams&, cudaStream_t);

}  // namespace b200fa
