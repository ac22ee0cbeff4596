// Exact-fp32 SIMT attention kernels (forward and backward).
//
// These serve fp32 tensors where fp32_sm100.cu does not, at head dimension 128: the backward, the forward ahead of it, and
// forwards over few keys.  All products and sums are fp32 FMAs; the softmax
// uses exp2f on scale*log2(e)-scaled scores, the same formulation as the tensor-core path
// (reference math: torch_mojo_backend/eager_flash_attention/fa4_fwd_kernel.mojo:650-861 and
// fa4_bwd_kernel.mojo:1-44, 810-980).  They are templated on the storage type so the same
// code can also read 16-bit tensors, which the tests use as an on-device cross-check of the
// tcgen05 kernels at sizes where a CPU oracle would take minutes.
//
// Tiling.  A block owns BM "row" positions (query rows in the forward and the dQ kernel, key rows in
// the dK/dV kernel) and walks the other sequence in tiles of 64 "column" positions.  The 16 x TY
// threads each own TM rows (groups of four neighbours: 4ty + i, and 4ty + 4TY + i) and the columns
// tx + 16j.  Two kinds of product:
//   * rows x columns (S, dP): both operands are (position, head dim) tiles, contracted over the head
//     dim.  A thread reads 16 bytes of each of its TM rows and 4 columns and issues packed two-wide
//     FMAs on them, even and odd head-dim elements in separate sums;
//   * rows x head dim (O, dQ, dK, dV): the score tile goes through shared memory as [column][row], so
//     that a thread reads its rows and its head-dim elements of one column as 16-byte vectors and
//     adds their outer product.
// Shared memory, not the fp32 pipe, bounds such a loop when a thread's tile is small: the 4x4 tile
// with scalar loads that preceded this one ran at 12 TFLOP/s.  With 16-byte loads the 8x4 loop alone
// measures 53 TFLOP/s (rows x columns) and 60-62 (rows x head dim); 4x4 44-48; the pipe's peak is 74.
// The 16-byte pieces of a row are XOR-permuted by the row's index, (row >> 2) & 7 for the resident
// tiles and row & 7 for the streamed ones, so that the rows one quarter-warp reads lie in different
// banks; a [column][row] tile has rows of BM + 4 floats for the same reason.
// Loads are asynchronous copies into the one buffer that each streamed tile has: a tile is fetched
// while the product that does not need it runs.
//
// One translation unit per storage type (simt.cu, simt_bf16.cu, simt_f16.cu): together they are most of the
// library's compile time.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "philox.cuh"
#include "ptx.cuh"

namespace b200fa {
namespace {

constexpr int kBN = 64;     // columns per step
constexpr int kTX = 16;     // threads across the columns / the head dim
constexpr int kTN = kBN / kTX;
constexpr float kLog2e = 1.4426950408889634f;

template <typename T>
__device__ __forceinline__ const T* row_ptr(const View4& t, int b, int h, int s) {
  return reinterpret_cast<const T*>(t.ptr) + (int64_t)b * t.sb + (int64_t)h * t.sh + (int64_t)s * t.ss;
}
template <typename T>
__device__ __forceinline__ T* row_ptr_mut(const View4& t, int b, int h, int s) {
  return reinterpret_cast<T*>(t.ptr) + (int64_t)b * t.sb + (int64_t)h * t.sh + (int64_t)s * t.ss;
}
template <typename T>
__device__ __forceinline__ float to_f32(T x);
template <>
__device__ __forceinline__ float to_f32<float>(float x) { return x; }
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }
template <>
__device__ __forceinline__ float to_f32<__half>(__half x) { return __half2float(x); }

// four consecutive elements as floats, and back (rounded to nearest)
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
  const uint2 w = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16),
                     __uint_as_float(w.y & 0xffff0000u));
}
__device__ __forceinline__ float4 load4(const __half* p) {
  const uint2 w = *reinterpret_cast<const uint2*>(p);
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&w.x));
  const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&w.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void store4(float* p, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
__device__ __forceinline__ void store4(__nv_bfloat16* p, float a, float b, float c, float d) {
  const __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}
__device__ __forceinline__ void store4(__half* p, float a, float b, float c, float d) {
  const __half2 lo = __floats2half2_rn(a, b), hi = __floats2half2_rn(c, d);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

// The shape of a block: TM rows per thread, TY threads down the rows.
template <int kTM, int kTY>
struct Shape {
  static constexpr int TM = kTM, TY = kTY;
  static constexpr int BM = TM * TY, NT = kTX * TY, LDX = BM + 4;
  // local row of a thread's i-th row
  static __device__ __forceinline__ int row(int ty, int i) { return 4 * ty + (i & 3) + (i >> 2) * 4 * TY; }
};

// `kRows` rows x kD columns to shared memory as fp32; rows at or past `S` are zero.  kShift: which
// bits of the row index permute its 16-byte pieces (2: resident tiles, 0: streamed tiles).
template <typename T, int kD, int kRows, int kNT, int kShift>
__device__ __forceinline__ void stage_tile(float* dst, const View4& t, int b, int h, int s0, int S) {
  const T* base = row_ptr<T>(t, b, h, 0);
  constexpr int kPieces = kD / 4;
  static_assert(kRows * kPieces % kNT == 0, "whole pieces per thread");
#pragma unroll
  for (int it = 0; it < kRows * kPieces / kNT; ++it) {
    const int idx = threadIdx.x + it * kNT;
    const int r = idx / kPieces, c = idx % kPieces;
    float* d = dst + r * kD + ((c ^ ((r >> kShift) & 7)) << 2);
    const bool inside = s0 + r < S;
    const T* src = base + (int64_t)(inside ? s0 + r : 0) * t.ss + c * 4;
    if constexpr (sizeof(T) == 4) {
      cp_async16(d, src, inside);
    } else {
      *reinterpret_cast<float4*>(d) = inside ? load4(src) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

// acc[i][j] = sum over the head dim of A[row i] * B[column j]
template <class S, int kD>
__device__ __forceinline__ void rows_by_cols(const float* A, const float* B, int tx, int ty, float (&acc)[S::TM][kTN]) {
  float2 a2[S::TM][kTN];
#pragma unroll
  for (int i = 0; i < S::TM; ++i)
#pragma unroll
    for (int j = 0; j < kTN; ++j) a2[i][j] = make_float2(0.f, 0.f);
  const float* ab = A + 4 * ty * kD;
  const float* bb = B + tx * kD;
#pragma unroll 8
  for (int c = 0; c < kD / 4; ++c) {
    float4 a[S::TM], w[kTN];
    const int ca = (c ^ (ty & 7)) << 2, cb = (c ^ (tx & 7)) << 2;
#pragma unroll
    for (int i = 0; i < S::TM; ++i) a[i] = *reinterpret_cast<const float4*>(ab + ca + ((i & 3) + (i >> 2) * 4 * S::TY) * kD);
#pragma unroll
    for (int j = 0; j < kTN; ++j) w[j] = *reinterpret_cast<const float4*>(bb + cb + j * kTX * kD);
#pragma unroll
    for (int i = 0; i < S::TM; ++i)
#pragma unroll
      for (int j = 0; j < kTN; ++j) {
        a2[i][j] = __ffma2_rn(make_float2(a[i].x, a[i].y), make_float2(w[j].x, w[j].y), a2[i][j]);
        a2[i][j] = __ffma2_rn(make_float2(a[i].z, a[i].w), make_float2(w[j].z, w[j].w), a2[i][j]);
      }
  }
#pragma unroll
  for (int i = 0; i < S::TM; ++i)
#pragma unroll
    for (int j = 0; j < kTN; ++j) acc[i][j] = a2[i][j].x + a2[i][j].y;
}

// acc[i][e] += sum over the 64 columns of X[column][row i] * W[column][element e]; element e of a
// thread is 4tx + e % 4 + 64 (e / 4)
template <class S, int kD>
__device__ __forceinline__ void rows_by_dim(const float* X, const float* W, int tx, int ty, float2 (&acc)[S::TM][kD / 32]) {
  const float* xb = X + 4 * ty;
#pragma unroll 8
  for (int k = 0; k < kBN; ++k) {
    float x[S::TM];
    float2 w[kD / 32];
#pragma unroll
    for (int i = 0; i < S::TM; i += 4) {
      const float4 v = *reinterpret_cast<const float4*>(xb + k * S::LDX + i * S::TY);
      x[i] = v.x; x[i + 1] = v.y; x[i + 2] = v.z; x[i + 3] = v.w;
    }
#pragma unroll
    for (int e = 0; e < kD / 64; ++e) {
      const float4 v = *reinterpret_cast<const float4*>(W + k * kD + ((tx ^ (k & 7)) << 2) + e * 64);
      w[2 * e] = make_float2(v.x, v.y);
      w[2 * e + 1] = make_float2(v.z, v.w);
    }
#pragma unroll
    for (int i = 0; i < S::TM; ++i)
#pragma unroll
      for (int e = 0; e < kD / 32; ++e) acc[i][e] = __ffma2_rn(make_float2(x[i], x[i]), w[e], acc[i][e]);
  }
}

// the thread's scores to the [column][row] tile
template <class S>
__device__ __forceinline__ void scores_to_shared(float* X, int tx, int ty, const float (&v)[S::TM][kTN]) {
#pragma unroll
  for (int j = 0; j < kTN; ++j)
#pragma unroll
    for (int i = 0; i < S::TM; i += 4)
      store4(X + (tx + kTX * j) * S::LDX + 4 * ty + i * S::TY, v[i][j], v[i + 1][j], v[i + 2][j], v[i + 3][j]);
}

// the thread's rows of an accumulator, times `mul[i]`, to the rows s0 + .. of a (B, H, S, D) tensor
template <class S, typename T, int kD>
__device__ __forceinline__ void store_rows(const View4& t, int b, int h, int s0, int n_rows, int tx, int ty,
                                           const float2 (&acc)[S::TM][kD / 32], const float (&mul)[S::TM]) {
#pragma unroll
  for (int i = 0; i < S::TM; ++i) {
    const int s = s0 + S::row(ty, i);
    if (s < n_rows) {
      T* row = row_ptr_mut<T>(t, b, h, s) + 4 * tx;
#pragma unroll
      for (int e = 0; e < kD / 64; ++e)
        store4(row + e * 64, acc[i][2 * e].x * mul[i], acc[i][2 * e].y * mul[i], acc[i][2 * e + 1].x * mul[i],
               acc[i][2 * e + 1].y * mul[i]);
    }
  }
}

template <int kD>
__device__ __forceinline__ float group_max(float v) {
#pragma unroll
  for (int o = kD / 2; o >= 1; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <int kD>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = kD / 2; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// bytes: `resident` tiles of BM rows, two streamed tiles, the [column][row] tile, keep bits, two statistics per column
template <class S, int kD>
constexpr int smem_bytes(int resident) {
  return (resident * S::BM * kD + 2 * kBN * kD + kBN * S::LDX) * 4 + S::BM * 8 + 2 * kBN * 4;
}

// Block index -> (row tile, head); the longest causal rows first over all heads, so that the last
// wave is made of short blocks
__device__ __forceinline__ void tile_and_head(int tiles, int heads, bool latest_first, int* tile, int* bh) {
  const int t = static_cast<int>(blockIdx.x) / heads;
  *bh = static_cast<int>(blockIdx.x) - t * heads;
  *tile = latest_first ? tiles - 1 - t : t;
}

// ------------------------------------------------------------------------------------------
// forward
// ------------------------------------------------------------------------------------------
template <class S, typename T, int kD, bool kDrop>
__global__ void __launch_bounds__(S::NT, 1) fwd_simt_kernel(const FwdParams p) {
  extern __shared__ __align__(16) float sm[];
  float* sQ = sm;
  float* sK = sQ + S::BM * kD;
  float* sV = sK + kBN * kD;
  float* sX = sV + kBN * kD;
  uint64_t* sKeep = reinterpret_cast<uint64_t*>(sX + kBN * S::LDX);   // one bit per column, a word per row
  const int tx = threadIdx.x % kTX, ty = threadIdx.x / kTX;
  int tile, bh;
  tile_and_head((p.Sq + S::BM - 1) / S::BM, p.B * p.Hq, p.causal, &tile, &bh);
  const int m0 = tile * S::BM;
  const int b = bh / p.Hq, h = bh - b * p.Hq;
  const int hk = h / (p.Hq / p.Hkv);
  const float c = p.scale_log2;

  float2 o[S::TM][kD / 32];
  float mrow[S::TM], lrow[S::TM];   // lrow: this thread's columns only, summed over the row at the end
#pragma unroll
  for (int i = 0; i < S::TM; ++i) {
    mrow[i] = -INFINITY;
    lrow[i] = 0.f;
#pragma unroll
    for (int e = 0; e < kD / 32; ++e) o[i][e] = make_float2(0.f, 0.f);
  }
  // query row i sees key column j iff j <= i + causal_off
  const int n_end = p.causal ? max(0, min(p.Sk, min(m0 + S::BM, p.Sq) + p.causal_off)) : p.Sk;
  stage_tile<T, kD, S::BM, S::NT, 2>(sQ, p.q, b, h, m0, p.Sq);
  if (n_end > 0) stage_tile<T, kD, kBN, S::NT, 0>(sK, p.k, b, hk, 0, p.Sk);
  cp_commit();
  for (int n0 = 0; n0 < n_end; n0 += kBN) {
    cp_wait<0>();
    __syncthreads();   // K is here; the last step is done with V and the score tile
    stage_tile<T, kD, kBN, S::NT, 0>(sV, p.v, b, hk, n0, p.Sk);
    cp_commit();
    if constexpr (kDrop) {
      for (int idx = threadIdx.x; idx < S::BM * 4; idx += S::NT)
        reinterpret_cast<uint16_t*>(sKeep)[idx] =
            static_cast<uint16_t>(dropout_bits16(p.drop, bh, m0 + (idx >> 2), (n0 >> 4) + (idx & 3)));
    }
    float s[S::TM][kTN];
    rows_by_cols<S, kD>(sQ, sK, tx, ty, s);
    __syncthreads();   // everyone is done with K
    if (n0 + kBN < n_end) stage_tile<T, kD, kBN, S::NT, 0>(sK, p.k, b, hk, n0 + kBN, p.Sk);
    cp_commit();
    const bool need_mask = n0 + kBN > p.Sk || (p.causal && n0 + kBN - 1 > m0 + p.causal_off);
#pragma unroll
    for (int i = 0; i < S::TM; ++i) {
      const int r = S::row(ty, i);
      if (need_mask) {
        const int last = p.causal ? min(m0 + r + p.causal_off, p.Sk - 1) : p.Sk - 1;
#pragma unroll
        for (int j = 0; j < kTN; ++j)
          if (n0 + tx + kTX * j > last) s[i][j] = -INFINITY;
      }
      float mx = s[i][0];
#pragma unroll
      for (int j = 1; j < kTN; ++j) mx = fmaxf(mx, s[i][j]);
      mx = group_max<kTX>(mx);
      float m_new = fmaxf(mrow[i], mx);
      if (m_new == -INFINITY) m_new = 0.f;
      const float corr = exp2f((mrow[i] - m_new) * c);
      float rs = 0.f;
#pragma unroll
      for (int j = 0; j < kTN; ++j) {
        s[i][j] = exp2f((s[i][j] - m_new) * c);
        rs += s[i][j];   // the row sum keeps every probability; only what multiplies V is dropped
      }
      if constexpr (kDrop) {
        const uint64_t keep = sKeep[r] >> tx;
#pragma unroll
        for (int j = 0; j < kTN; ++j)
          if (!((keep >> (kTX * j)) & 1u)) s[i][j] = 0.f;
      }
      lrow[i] = lrow[i] * corr + rs;
      mrow[i] = m_new;
#pragma unroll
      for (int e = 0; e < kD / 32; ++e) o[i][e] = __fmul2_rn(o[i][e], make_float2(corr, corr));
    }
    scores_to_shared<S>(sX, tx, ty, s);
    cp_wait<1>();
    __syncthreads();   // V and the probabilities are here
    rows_by_dim<S, kD>(sX, sV, tx, ty, o);
  }
  cp_wait<0>();
  float inv[S::TM];
#pragma unroll
  for (int i = 0; i < S::TM; ++i) {
    const float l = group_sum<kTX>(lrow[i]);
    // a row that saw no key at all (possible under a bottom-right aligned mask) is 0 with lse -inf
    inv[i] = l > 0.f ? (kDrop ? p.drop.inv_keep : 1.f) / l : 0.f;
    const int qr = m0 + S::row(ty, i);
    if (tx == 0 && qr < p.Sq)
      p.lse[((int64_t)b * p.Hq + h) * p.Sq + qr] = l > 0.f ? mrow[i] * p.scale + logf(l) : -INFINITY;
  }
  store_rows<S, T, kD>(p.out, b, h, m0, p.Sq, tx, ty, o, inv);
}

// ------------------------------------------------------------------------------------------
// backward, part 1: dK and dV.  One block per (key tile, kv head, batch); loops over the query
// heads of the group and over the query tiles at or below the diagonal.  Rows are keys, columns
// are queries.
//   P = exp2(S*c - lse*log2e),  dV += P^T dO,  dS = P * (dP - dpsum),  dK += scale * dS^T Q
// ------------------------------------------------------------------------------------------
template <class S, typename T, int kD, bool kDrop>
__global__ void __launch_bounds__(S::NT, 1) bwd_dkdv_simt_kernel(const BwdParams p) {
  extern __shared__ __align__(16) float sm[];
  float* sK = sm;
  float* sV = sK + S::BM * kD;
  float* sQ = sV + S::BM * kD;
  float* sdO = sQ + kBN * kD;
  float* sX = sdO + kBN * kD;            // P, then dS
  uint16_t* sKeep = reinterpret_cast<uint16_t*>(sX + kBN * S::LDX);      // [query][key / 16]
  float* sLse = reinterpret_cast<float*>(sKeep) + S::BM * 2;             // [64]
  float* sDps = sLse + kBN;                                              // [64]
  const int tx = threadIdx.x % kTX, ty = threadIdx.x / kTX;
  int tile, bh;
  tile_and_head((p.Sk + S::BM - 1) / S::BM, p.B * p.Hkv, false, &tile, &bh);
  const int n0 = tile * S::BM;
  const int b = bh / p.Hkv, hk = bh - b * p.Hkv;
  const int group = p.Hq / p.Hkv;
  const float c = p.scale_log2;

  float2 dk[S::TM][kD / 32], dv[S::TM][kD / 32];
#pragma unroll
  for (int i = 0; i < S::TM; ++i)
#pragma unroll
    for (int e = 0; e < kD / 32; ++e) dk[i][e] = dv[i][e] = make_float2(0.f, 0.f);

  const int m_begin = p.causal ? max(0, n0 - p.causal_off) / kBN * kBN : 0;   // first tile with a query that sees a key
  const int per_head = max(0, (p.S - m_begin + kBN - 1) / kBN);
  const int steps = group * per_head;
  stage_tile<T, kD, S::BM, S::NT, 2>(sK, p.k, b, hk, n0, p.Sk);
  stage_tile<T, kD, S::BM, S::NT, 2>(sV, p.v, b, hk, n0, p.Sk);
  if (steps > 0) stage_tile<T, kD, kBN, S::NT, 0>(sdO, p.dout, b, hk * group, m_begin, p.S);
  cp_commit();
  for (int step = 0; step < steps; ++step) {
    const int h = hk * group + step / per_head;
    const int m0 = m_begin + step % per_head * kBN;
    cp_wait<0>();
    __syncthreads();   // dO is here; the last step is done with Q and the score tile
    stage_tile<T, kD, kBN, S::NT, 0>(sQ, p.q, b, h, m0, p.S);
    cp_commit();
    if (threadIdx.x < kBN) {
      const int qr = m0 + threadIdx.x;
      float l2 = INFINITY;   // rows past the end, and rows that saw no key (lse = -inf): P = 0
      if (qr < p.S) {
        const float l = p.lse[((int64_t)b * p.Hq + h) * p.S + qr];
        if (l != -INFINITY) l2 = l * kLog2e;
      }
      sLse[threadIdx.x] = l2;
      sDps[threadIdx.x] = (qr < p.S) ? p.dpsum[((int64_t)b * p.Hq + h) * p.Spad + qr] : 0.f;
    }
    if constexpr (kDrop) {
      for (int idx = threadIdx.x; idx < kBN * S::BM / 16; idx += S::NT)
        sKeep[idx] = static_cast<uint16_t>(
            dropout_bits16(p.drop, b * p.Hq + h, m0 + idx / (S::BM / 16), (n0 >> 4) + idx % (S::BM / 16)));
    }
    float s[S::TM][kTN], dp[S::TM][kTN];
    rows_by_cols<S, kD>(sV, sdO, tx, ty, dp);
    cp_wait<0>();
    __syncthreads();   // Q and the statistics are here
    rows_by_cols<S, kD>(sK, sQ, tx, ty, s);
    const bool need_mask = n0 + S::BM > p.Sk || m0 + kBN > p.S || (p.causal && n0 + S::BM - 1 > m0 + p.causal_off);
#pragma unroll
    for (int j = 0; j < kTN; ++j) {
      const int ql = tx + kTX * j, qr = m0 + ql;
      const float l2 = sLse[ql], dps = sDps[ql];
#pragma unroll
      for (int i = 0; i < S::TM; ++i) {
        const int kc = n0 + S::row(ty, i);
        float pv = exp2f(s[i][j] * c - l2);
        if (need_mask && (kc >= p.Sk || qr >= p.S || (p.causal && kc > qr + p.causal_off))) pv = 0.f;
        float dm = 1.f;   // dropout multiplier of this entry: 0 or 1 / (1 - p)
        if constexpr (kDrop) {
          const int r = S::row(ty, i);
          dm = ((sKeep[ql * (S::BM / 16) + (r >> 4)] >> (r & 15)) & 1u) ? p.drop.inv_keep : 0.f;
        }
        dp[i][j] = pv * (dp[i][j] * dm - dps);   // dS
        s[i][j] = pv * dm;
      }
    }
    scores_to_shared<S>(sX, tx, ty, s);
    __syncthreads();
    rows_by_dim<S, kD>(sX, sdO, tx, ty, dv);     // dV[key] += P[query][key] dO[query]
    __syncthreads();   // everyone is done with P and dO
    if (step + 1 < steps)
      stage_tile<T, kD, kBN, S::NT, 0>(sdO, p.dout, b, hk * group + (step + 1) / per_head,
                                       m_begin + (step + 1) % per_head * kBN, p.S);
    cp_commit();
    scores_to_shared<S>(sX, tx, ty, dp);
    __syncthreads();
    rows_by_dim<S, kD>(sX, sQ, tx, ty, dk);      // dK[key] += dS[query][key] Q[query]
  }
  cp_wait<0>();
  float one[S::TM], scale[S::TM];
#pragma unroll
  for (int i = 0; i < S::TM; ++i) {
    one[i] = 1.f;
    scale[i] = p.scale;
  }
  store_rows<S, T, kD>(p.dk, b, hk, n0, p.Sk, tx, ty, dk, scale);
  store_rows<S, T, kD>(p.dv, b, hk, n0, p.Sk, tx, ty, dv, one);
}

// ------------------------------------------------------------------------------------------
// backward, part 2: dQ.  One block per (query tile, q head, batch); loops over the key tiles up
// to the diagonal.  dQ = scale * dS K.  Deterministic: no atomics.
// ------------------------------------------------------------------------------------------
template <class S, typename T, int kD, bool kDrop>
__global__ void __launch_bounds__(S::NT, 1) bwd_dq_simt_kernel(const BwdParams p) {
  extern __shared__ __align__(16) float sm[];
  float* sQ = sm;
  float* sdO = sQ + S::BM * kD;
  float* sK = sdO + S::BM * kD;
  float* sV = sK + kBN * kD;
  float* sX = sV + kBN * kD;             // dS
  uint64_t* sKeep = reinterpret_cast<uint64_t*>(sX + kBN * S::LDX);   // one bit per column, a word per row
  const int tx = threadIdx.x % kTX, ty = threadIdx.x / kTX;
  int tile, bh;
  tile_and_head((p.S + S::BM - 1) / S::BM, p.B * p.Hq, p.causal, &tile, &bh);
  const int m0 = tile * S::BM;
  const int b = bh / p.Hq, h = bh - b * p.Hq;
  const int hk = h / (p.Hq / p.Hkv);
  const float c = p.scale_log2;

  float lse2[S::TM], dps[S::TM];
  float2 dq[S::TM][kD / 32];
#pragma unroll
  for (int i = 0; i < S::TM; ++i) {
    const int qr = m0 + S::row(ty, i);
    lse2[i] = INFINITY;
    if (qr < p.S) {
      const float l = p.lse[((int64_t)b * p.Hq + h) * p.S + qr];
      if (l != -INFINITY) lse2[i] = l * kLog2e;
    }
    dps[i] = (qr < p.S) ? p.dpsum[((int64_t)b * p.Hq + h) * p.Spad + qr] : 0.f;
#pragma unroll
    for (int e = 0; e < kD / 32; ++e) dq[i][e] = make_float2(0.f, 0.f);
  }
  const int n_end = p.causal ? max(0, min(p.Sk, min(m0 + S::BM, p.S) + p.causal_off)) : p.Sk;
  stage_tile<T, kD, S::BM, S::NT, 2>(sQ, p.q, b, h, m0, p.S);
  stage_tile<T, kD, S::BM, S::NT, 2>(sdO, p.dout, b, h, m0, p.S);
  if (n_end > 0) stage_tile<T, kD, kBN, S::NT, 0>(sV, p.v, b, hk, 0, p.Sk);
  cp_commit();
  for (int n0 = 0; n0 < n_end; n0 += kBN) {
    cp_wait<0>();
    __syncthreads();   // V is here; the last step is done with K and the score tile
    stage_tile<T, kD, kBN, S::NT, 0>(sK, p.k, b, hk, n0, p.Sk);
    cp_commit();
    if constexpr (kDrop) {
      for (int idx = threadIdx.x; idx < S::BM * 4; idx += S::NT)
        reinterpret_cast<uint16_t*>(sKeep)[idx] =
            static_cast<uint16_t>(dropout_bits16(p.drop, bh, m0 + (idx >> 2), (n0 >> 4) + (idx & 3)));
    }
    float s[S::TM][kTN], dp[S::TM][kTN];
    rows_by_cols<S, kD>(sdO, sV, tx, ty, dp);
    cp_wait<0>();
    __syncthreads();   // K is here; everyone is done with V
    if (n0 + kBN < n_end) stage_tile<T, kD, kBN, S::NT, 0>(sV, p.v, b, hk, n0 + kBN, p.Sk);
    cp_commit();
    rows_by_cols<S, kD>(sQ, sK, tx, ty, s);
    const bool need_mask = n0 + kBN > p.Sk || m0 + S::BM > p.S || (p.causal && n0 + kBN - 1 > m0 + p.causal_off);
#pragma unroll
    for (int i = 0; i < S::TM; ++i) {
      const int r = S::row(ty, i), qr = m0 + r;
      uint64_t keep = 0;
      if constexpr (kDrop) keep = sKeep[r] >> tx;
#pragma unroll
      for (int j = 0; j < kTN; ++j) {
        const int kc = n0 + tx + kTX * j;
        float pv = exp2f(s[i][j] * c - lse2[i]);
        if (need_mask && (kc >= p.Sk || qr >= p.S || (p.causal && kc > qr + p.causal_off))) pv = 0.f;
        float dm = 1.f;
        if constexpr (kDrop) dm = ((keep >> (kTX * j)) & 1u) ? p.drop.inv_keep : 0.f;
        s[i][j] = pv * (dp[i][j] * dm - dps[i]);
      }
    }
    scores_to_shared<S>(sX, tx, ty, s);
    __syncthreads();
    rows_by_dim<S, kD>(sX, sK, tx, ty, dq);      // dQ[query] += dS[query][key] K[key]
  }
  cp_wait<0>();
  float scale[S::TM];
#pragma unroll
  for (int i = 0; i < S::TM; ++i) scale[i] = p.scale;
  store_rows<S, T, kD>(p.dq, b, h, m0, p.S, tx, ty, dq, scale);
}

// dpsum[b,h,s] = sum_d dO * O (fp32), one warp per row.
template <typename T>
__global__ void dpsum_simt_kernel(const BwdParams p) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int64_t rows = (int64_t)p.B * p.Hq * p.S;
  if (warp >= rows) return;
  const int s = (int)(warp % p.S);
  const int h = (int)((warp / p.S) % p.Hq);
  const int b = (int)(warp / ((int64_t)p.S * p.Hq));
  const T* o = row_ptr<T>(p.out, b, h, s);
  const T* d = row_ptr<T>(p.dout, b, h, s);
  float acc = 0.f;
  for (int i = lane; i < p.D; i += 32) acc = fmaf(to_f32<T>(o[i]), to_f32<T>(d[i]), acc);
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (lane == 0) p.dpsum[((int64_t)b * p.Hq + h) * p.Spad + s] = acc;
}

template <typename Kernel, typename Params>
cudaError_t launch(Kernel kern, int64_t blocks, int threads, int smem, cudaStream_t stream, const Params& p) {
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  kern<<<static_cast<unsigned>(blocks), threads, smem, stream>>>(p);
  return cudaGetLastError();
}

// Which shape.  Tall: at D = 64 an 8x4 tile a thread and 128 threads, at D = 128 (where the
// accumulators of 8 rows spill) 4x4 and 256 threads; both 64 rows a block.  Short: 4x4, 128 threads
// and 32 rows a block, for problems whose tall blocks leave the chip partly idle: fewer than three
// per SM.  Measured (us, B200, causal S = 1024, forward / backward, Short against Tall):
//   D=64:  192 tall blocks 62 / 201 against 79 / 265, 384: 104 / 335 against 104 / 354,
//          480: 125 / 409 against 113 / 379, 768: 195 / 641 against 165 / 566
//   D=128: 64 tall blocks 74 / 244 against 125 / 406, 192: 108 / 355 against 125 / 410,
//          384: 180 / 589 against 189 / 623, 1024: 479 / 1655 against 469 / 1547
// With the 4x4 scalar kernels that preceded both: 416 / 1361 at D = 64, 768 blocks.
template <int kD> using Tall = Shape<kD == 64 ? 8 : 4, kD == 64 ? 8 : 16>;
using Short = Shape<4, 8>;
bool short_blocks(int64_t heads, int rows) { return heads * ((rows + 63) / 64) < 3 * 148; }

template <class S, typename T, int kD>
cudaError_t launch_fwd_s(const FwdParams& p, cudaStream_t stream) {
  const int64_t blocks = (int64_t)p.B * p.Hq * ((p.Sq + S::BM - 1) / S::BM);
  constexpr int smem = smem_bytes<S, kD>(1);
  return p.drop.threshold != 0 ? launch(fwd_simt_kernel<S, T, kD, true>, blocks, S::NT, smem, stream, p)
                               : launch(fwd_simt_kernel<S, T, kD, false>, blocks, S::NT, smem, stream, p);
}

template <typename T, int kD>
cudaError_t launch_fwd_t(const FwdParams& p, cudaStream_t stream) {
  return short_blocks((int64_t)p.B * p.Hq, p.Sq) ? launch_fwd_s<Short, T, kD>(p, stream)
                                                     : launch_fwd_s<Tall<kD>, T, kD>(p, stream);
}

template <class S, typename T, int kD>
cudaError_t launch_dkdv_s(const BwdParams& p, cudaStream_t stream) {
  const int64_t blocks = (int64_t)p.B * p.Hkv * ((p.Sk + S::BM - 1) / S::BM);
  constexpr int smem = smem_bytes<S, kD>(2);
  return p.drop.threshold != 0 ? launch(bwd_dkdv_simt_kernel<S, T, kD, true>, blocks, S::NT, smem, stream, p)
                               : launch(bwd_dkdv_simt_kernel<S, T, kD, false>, blocks, S::NT, smem, stream, p);
}

template <class S, typename T, int kD>
cudaError_t launch_dq_s(const BwdParams& p, cudaStream_t stream) {
  const int64_t blocks = (int64_t)p.B * p.Hq * ((p.S + S::BM - 1) / S::BM);
  constexpr int smem = smem_bytes<S, kD>(2);
  return p.drop.threshold != 0 ? launch(bwd_dq_simt_kernel<S, T, kD, true>, blocks, S::NT, smem, stream, p)
                               : launch(bwd_dq_simt_kernel<S, T, kD, false>, blocks, S::NT, smem, stream, p);
}

template <typename T, int kD>
cudaError_t launch_bwd_t(const BwdParams& p, cudaStream_t stream) {
  const int64_t rows = (int64_t)p.B * p.Hq * p.S;
  dpsum_simt_kernel<T><<<(unsigned)((rows * 32 + 255) / 256), 256, 0, stream>>>(p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  e = short_blocks((int64_t)p.B * p.Hkv, p.Sk) ? launch_dkdv_s<Short, T, kD>(p, stream)
                                                   : launch_dkdv_s<Tall<kD>, T, kD>(p, stream);
  if (e != cudaSuccess) return e;
  return short_blocks((int64_t)p.B * p.Hq, p.S) ? launch_dq_s<Short, T, kD>(p, stream)
                                                    : launch_dq_s<Tall<kD>, T, kD>(p, stream);
}

}  // namespace

template <typename T>
cudaError_t simt_fwd(const FwdParams& p, cudaStream_t stream) {
  return p.D == 64 ? launch_fwd_t<T, 64>(p, stream) : launch_fwd_t<T, 128>(p, stream);
}

template <typename T>
cudaError_t simt_bwd(const BwdParams& p, cudaStream_t stream) {
  return p.D == 64 ? launch_bwd_t<T, 64>(p, stream) : launch_bwd_t<T, 128>(p, stream);
}

}  // namespace b200fa
