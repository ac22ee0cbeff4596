// Shared declarations between the host entry points (api.cu) and the kernel translation
// units.  Everything here is internal to the library; the public surface is include/b200fa.h.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200fa {

// A validated (B, H, S, D) view: base pointer plus element strides (D stride is 1).
struct View4 {
  void* ptr;
  int64_t sb, sh, ss;
};

// Dropout: element (b, h, i, j) of the attention matrix is kept when its byte of a
// Philox4x32-10 stream keyed by `seed` is >= `threshold` (see philox.cuh); kept probabilities
// are multiplied by `inv_keep` = 1 / (1 - p).  threshold == 0 means no dropout.
struct DropoutParams {
  uint64_t seed;
  uint64_t offset;
  uint32_t threshold;  // 0..255: bytes below it are dropped
  float inv_keep;
};

struct FwdParams {
  View4 q, k, v, out;
  float* lse;        // (B, Hq, Sq) fp32 contiguous
  int B, Hq, Hkv, Sq, Sk, D;
  int causal;        // 0: no mask; otherwise query row i sees key column j iff j <= i + causal_off
  int causal_off;    // 0 (top-left aligned diagonal) or Sk - Sq (bottom-right aligned)
  float scale;       // softmax scale
  float scale_log2;  // scale * log2(e)
  uint32_t* status;  // optional device status word
  int64_t whole_heads;    // batch * query heads of the problem this one is a piece of (its own, if it is whole)
  int tiles_per_cta;      // forward kernel shape: 0 = chosen by the launcher, 1 or 2 = forced
  long long wait_budget;  // SM cycles any single internal wait may take before the kernel gives up
  DropoutParams drop;
};

struct BwdParams {
  View4 q, k, v, out, dout, dq, dk, dv;
  const float* lse;  // (B, Hq, S) fp32 contiguous (natural log)
  float* dpsum;      // workspace: (B, Hq, Spad) rowsum(dO * O)   (the tensor-core route stores both
  float* lse_log2;   // workspace: (B, Hq, Spad) lse * log2(e)     statistics negated, the SIMT route as is)
  int B, Hq, Hkv, S, Sk, Spad, D;   // S: query rows (Spad: padded to 128); Sk: key rows
  int causal;
  int causal_off;
  float scale;
  float scale_log2;
  uint32_t* status;
  long long wait_budget;
  int parts;  // bit 0 preprocess, bit 1 dK/dV kernel, bit 2 dQ kernel (7 = the whole backward)
  DropoutParams drop;
};

// Split-KV forward for short query blocks (decode): partial (max, sum, O) per key split.
struct SplitKvParams {
  View4 q, k, v, out;
  float* lse;
  float* part_o;    // workspace: (B, Hq, Sq, nsplit, D) fp32
  float* part_ml;   // workspace: (B, Hq, Sq, nsplit, 2) fp32: running max (log2 domain), row sum
  unsigned* counters;   // workspace: (B, Hkv) splits finished so far, zeroed before the launch
  int B, Hq, Hkv, Sq, Sk, D;
  int causal, causal_off;
  int nsplit, split_len;   // keys per split (a multiple of 64)
  float scale, scale_log2;
};

constexpr int kSplitkvCluster = 16;   // splits of a KV head that may merge as a cluster

// dtype tags shared with the C header
constexpr int kF32 = 0, kBF16 = 1, kF16 = 2;

// Launchers implemented in the kernel translation units.  Each returns a cudaError_t and
// adds the number of kernels it enqueued to *launches.
cudaError_t launch_fwd_sm100(const FwdParams& p, int dtype, cudaStream_t stream, int* launches);
int fwd_splits(const FwdParams& p);   // CTAs that share a query unit's K/V blocks in launch_fwd_sm100 (host only)
cudaError_t launch_fwd_simt(const FwdParams& p, int dtype, cudaStream_t stream, int* launches);
cudaError_t launch_fwd_fp32(const FwdParams& p, cudaStream_t stream, int* launches);   // fp32 on the tensor cores
cudaError_t launch_bwd_fp32(const BwdParams& p, cudaStream_t stream, int* launches);   // ... head dim 64
cudaError_t launch_fwd_splitkv(const SplitKvParams& p, int dtype, cudaStream_t stream, int* launches);
cudaError_t launch_bwd_sm100(const BwdParams& p, int dtype, cudaStream_t stream, int* launches);
cudaError_t launch_bwd_simt(const BwdParams& p, int dtype, cudaStream_t stream, int* launches);
// A one-warp kernel whose only job is to wait, with `budget` SM cycles, on a barrier nobody
// arrives at: exercises the bounded-wait give-up path without touching the attention kernels.
cudaError_t launch_wait_timeout_selftest(uint32_t* status, long long budget, cudaStream_t stream, int* launches);

// In the dK/dV kernels, by the threads that read the row statistics: waits for the kernel that wrote them and lets the dQ
// kernel start.  The dQ kernel does not wait for that one itself: it starts when every block has been here, and the fence
// orders what this thread has been shown ahead of that.  It reads the statistics from L2 (__ldcg), never through an L1
// line that may be older.
__device__ __forceinline__ void let_the_dq_kernel_start() {
  cudaGridDependencySynchronize();
  __threadfence();
  cudaTriggerProgrammaticLaunchCompletion();
}

// A launch that, if `early`, may start as soon as every block of the kernel ahead of it on the stream has allowed it.
template <typename... Params, typename... Args>
cudaError_t launch_early(void (*kern)(Params...), dim3 grid, int threads, int smem, cudaStream_t stream, bool early, Args... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(static_cast<unsigned>(threads));
  cfg.dynamicSmemBytes = static_cast<size_t>(smem);
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

// Encodes a 4-D tiled tensor map over a (B,H,S,D) view of 16-bit elements with a
// {64 x box_rows x 1 x 1} box and 128-byte swizzle.  Returns false if the driver entry
// point is unavailable or the encode fails.
bool encode_map_16bit(CUtensorMap* map, const View4& t, int B, int H, int S, int D, int box_rows, bool bf16);

}  // namespace b200fa
