// Attention on fp32 tensors through the bf16 tensor cores of sm_100a, at fp32 precision.
//
// An fp32 value is the exact sum of three bf16 values (24 bits of significand, eight each): x = h + m + l, h by
// truncation (it cannot overflow), m by rounding (l then has either sign, and so has what is left out below).  A product of two fp32 matrices is then six bf16 products,
//   l h' + h l' + m m' + m h' + h m' + h h',
// each exact in the tensor core and summed in fp32; what is left out (m l', l m', l l') is below 2^-22
// of |x x'| and zero on average.  tcgen05 truncates its accumulator after every 16 terms, always towards zero, so a
// long running sum would drift: the products are therefore issued smallest first, a tile product
// starts from zero, and the sum over the tiles of a row (O, dQ, dK, dV) is kept in registers and added to
// with rounding to nearest.  A single product is up to 2.0e-7 of itself off, where an FMA rounds to 6e-8; the long sums,
// which decide, are nearer to float64 than those of the fp32 FMA kernels (simt.cuh): at launch_fwd_fp32.
// Probabilities below 2^-126 of a row's largest are zero (ex2.approx.ftz).
// (The first part rounded to nearest too leaves out a quarter as much: errors 1-3 % smaller, kernels 1-13 % slower.)
//
// Same math and masks as simt.cuh (reference: torch_mojo_backend/eager_flash_attention/
// fa4_fwd_kernel.mojo:650-861, fa4_bwd_kernel.mojo:1-44, 810-980).  A CTA owns 128 resident rows and
// walks the other sequence in tiles of 64:
//   warps 0-7   math: thread <-> (resident row = TMEM lane, half of the 64 columns)
//   warps 8-11  converters: fp32 rows from global memory, split into three swizzled bf16 tiles in a
//               ring slot of shared memory
//   warp  12    issues the MMAs
// A 128x64 product over 64 elements is 24 MMAs of 128x64x16 (32 cycles each with the A operand in tensor memory, 48
// from shared memory), against ~14000 cycles of fp32 FMAs as measured.  No unit is the bound: the tensor pipe is busy 39 %
// (forward), 57 % (dK/dV) and 52 % (dQ) of the active cycles at B4 H12 S1024 D64, issue slots 36-45 %.  One CTA fits an SM, and
// what it waits for is its own chain of products, exponentials, splits and arrivals, two to three tiles deep.
//
// A product with an infinity cannot be split (inf * 0 is NaN): a CTA one of whose results is not finite computes its
// rows again with fp32 FMAs before it leaves, so that infinities spread as through fp32 products (fma_rows below).
#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "philox.cuh"
#include "ptx.cuh"

namespace b200fa {
namespace {

constexpr int kBM = 128;        // resident rows
constexpr int kBN = 64;         // rows of a streamed tile
constexpr int kThreads = 512;
constexpr int kMathWarps = 8, kConvWarp0 = 8, kConvWarps = 4, kMmaWarp = 12;
constexpr int kRegMath = 176, kRegConv = 104, kRegRest = 56;   // 256 * 176 + 128 * (104 + 56) = 512 * 128
constexpr int kBoxBytes = kBN * 128;   // 64 rows x 64 16-bit columns, 128-byte swizzle
constexpr float kLog2e = 1.4426950408889634f;

// A streamed tile in shared memory: [plane h, m, l][64-column box][row][128 B]
template <int kD>
struct TileCfg {
  static constexpr int kPlane = kBN * kD * 2, kBytes = 3 * kPlane, kBoxes = kD / 64;
};

// the products of the planes, smallest first: l h', h l', m m', m h', h m', h h' (a hex digit each, from the right)
constexpr uint32_t kPlanesA = 0x001102, kPlanesB = 0x010120;
__device__ __forceinline__ int plane_of(uint32_t planes, int t) { return (planes >> (4 * t)) & 3; }

#define B200FA_WAIT(bar, parity, site) \
  if (!mbar_wait((bar), (parity), abort_flag, p.status, (site), p.wait_budget)) goto teardown
#define B200FA_WAIT_WARP(bar, parity, site) \
  if (!mbar_wait_warp((bar), (parity), abort_flag, p.status, (site), p.wait_budget)) goto teardown

// The accumulator loses what does not fit towards zero, so scores come out short by a constant share on average:
// 6.9e-8 of them at D = 64 (four steps of full size) and 1.15e-7 at D = 128 (eight), measured as the slope of the
// error of lse over the mean score.  The resident operand of the scores is raised by as much, in its smallest plane
// (one ulp of it is too coarse); without that lse is 10 to 100 % further from float64 than the fp32 FMA kernels leave it.
// It fits scores whose 16-term steps look alike.  Where one channel outweighs the others or all terms are large, lse is 1.1 to
// 3.0 times as far from float64 as the FMA kernels leave it, still within an ulp (9e-8 of its value); out is nearer even so.
template <int kD>
constexpr float kLift = kD == 64 ? 6.9e-8f : 1.15e-7f;

// x0, x1 -> one word of each plane (lower half: x0)
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l, float lift = 0.f) {
  const float2 one = make_float2(-1.f, -1.f);
  const uint32_t u0 = __float_as_uint(x0), u1 = __float_as_uint(x1);
  h = __byte_perm(u0, u1, 0x7632);
  const float2 r = __ffma2_rn(make_float2(__uint_as_float(u0 & 0xffff0000u), __uint_as_float(u1 & 0xffff0000u)), one,
                              make_float2(x0, x1));
  const uint32_t v0 = __float_as_uint(r.x) + 0x8000u, v1 = __float_as_uint(r.y) + 0x8000u;
  m = __byte_perm(v0, v1, 0x7632);
  float2 t = __ffma2_rn(make_float2(__uint_as_float(v0 & 0xffff0000u), __uint_as_float(v1 & 0xffff0000u)), one, r);
  if (lift != 0.f) {
    t = __ffma2_rn(make_float2(x0, x1), make_float2(lift, lift), t);
    l = pack2<true>(t.x, t.y);   // (by the conversion: a NaN stays one, whose payload may be in bits that h does not have)
  } else {
    l = __byte_perm(__float_as_uint(t.x), __float_as_uint(t.y), 0x7632);   // (eight bits are left: exact)
  }
}

// are all of them finite (a multiple of zero of any other value is NaN)
template <int kN>
__device__ __forceinline__ bool all_finite(const float (&x)[kN]) {
  float2 seen = make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < kN / 2; ++i) seen = __ffma2_rn(make_float2(x[2 * i], x[2 * i + 1]), make_float2(0.f, 0.f), seen);
  return seen.x == 0.f && seen.y == 0.f;
}

__device__ __forceinline__ const float* row_ptr(const View4& t, int b, int h, int s) {
  return reinterpret_cast<const float*>(t.ptr) + (int64_t)b * t.sb + (int64_t)h * t.sh + (int64_t)s * t.ss;
}

// One box (64 rows x 64 columns) in two steps, so that the loads of the next one are in flight while this
// one is split: 128 threads, four 8-element pieces each.
__device__ __forceinline__ void load_box(float4 (&v)[8], const View4& t, int b, int h, int row0, int rows, int col0, int tid) {
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int idx = tid + it * 128, r = idx >> 3, c = idx & 7;
    v[2 * it] = v[2 * it + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row0 + r < rows) {
      const float4* src = reinterpret_cast<const float4*>(row_ptr(t, b, h, row0 + r) + col0 + c * 8);
      v[2 * it] = src[0];
      v[2 * it + 1] = src[1];
    }
  }
}
// `plane_bytes`: distance of the planes; rows r0 + .. of the box
__device__ __forceinline__ void store_piece(uint8_t* box, int plane_bytes, int r, int c, float4 x, float4 y, float lift = 0.f) {
  uint4 h, m, l;
  split2(x.x, x.y, h.x, m.x, l.x, lift);
  split2(x.z, x.w, h.y, m.y, l.y, lift);
  split2(y.x, y.y, h.z, m.z, l.z, lift);
  split2(y.z, y.w, h.w, m.w, l.w, lift);
  uint8_t* d = box + r * 128 + ((c ^ (r & 7)) << 4);
  *reinterpret_cast<uint4*>(d) = h;
  *reinterpret_cast<uint4*>(d + plane_bytes) = m;
  *reinterpret_cast<uint4*>(d + 2 * plane_bytes) = l;
}
__device__ __forceinline__ void store_box(const float4 (&v)[8], uint8_t* box, int plane_bytes, int tid) {
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int idx = tid + it * 128;
    store_piece(box, plane_bytes, idx >> 3, idx & 7, v[2 * it], v[2 * it + 1]);
  }
}

// This thread's half of its resident row to the three planes of a TMEM A operand (kD / 2 columns each)
template <int kD>
__device__ __forceinline__ void row_to_tmem(uint32_t taddr, const View4& t, int b, int h, int row, int rows, int half,
                                            float lift) {
#pragma unroll
  for (int part = 0; part < kD / 64; ++part) {
    uint32_t w[3][16];
    const float4* src = reinterpret_cast<const float4*>(row_ptr(t, b, h, row < rows ? row : 0) + half * (kD / 2) + part * 32);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 v = row < rows ? src[i] : make_float4(0.f, 0.f, 0.f, 0.f);
      split2(v.x, v.y, w[0][2 * i], w[1][2 * i], w[2][2 * i], lift);
      split2(v.z, v.w, w[0][2 * i + 1], w[1][2 * i + 1], w[2][2 * i + 1], lift);
    }
#pragma unroll
    for (int pl = 0; pl < 3; ++pl) tmem_st16(taddr + pl * (kD / 2) + half * (kD / 4) + part * 16, w[pl]);
  }
}

// 32 values of this thread's row to the three planes (32 columns each) of a 64-column TMEM A operand
__device__ __forceinline__ void values_to_tmem(uint32_t taddr, const float (&x)[32], int half) {
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    uint32_t w[3][8];
#pragma unroll
    for (int i = 0; i < 8; ++i) split2(x[part * 16 + 2 * i], x[part * 16 + 2 * i + 1], w[0][i], w[1][i], w[2][i]);
#pragma unroll
    for (int pl = 0; pl < 3; ++pl) tmem_st8(taddr + pl * 32 + half * 16 + part * 8, w[pl]);
  }
}

// acc[0 .. 32 kChunks) = acc * mul + the columns of the tile product
template <int kChunks>
__device__ __forceinline__ void add_part(float (&acc)[32 * kChunks], uint32_t taddr, float mul) {
  const float2 mul2 = make_float2(mul, mul);
#pragma unroll
  for (int ch = 0; ch < kChunks; ++ch) {
    float f[32];
    tmem_ld32(taddr + ch * 32, reinterpret_cast<uint32_t*>(f));
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float2 a = __ffma2_rn(make_float2(acc[ch * 32 + 2 * i], acc[ch * 32 + 2 * i + 1]), mul2, make_float2(f[2 * i], f[2 * i + 1]));
      acc[ch * 32 + 2 * i] = a.x;
      acc[ch * 32 + 2 * i + 1] = a.y;
    }
  }
}

// By the whole MMA warp.
// d[128 x 64] = A[128 x kD] (three planes in TMEM) * streamed tile[64 x kD]^T
template <int kD>
__device__ __forceinline__ void issue_cols_ts(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t b_hi) {
  constexpr uint32_t idesc = umma_idesc(true, false, false, kBM, kBN);
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    const uint32_t at = a + plane_of(kPlanesA, t) * (kD / 2), bt = b_lo + plane_of(kPlanesB, t) * umma_off(TileCfg<kD>::kPlane);
#pragma unroll
    for (int kk = 0; kk < kD / 16; ++kk)
      umma_ts_elect(d, at + kk * 8, bt + umma_off((kk >> 2) * kBoxBytes + (kk & 3) * 32), b_hi, idesc, kk > 0 || t > 0);
  }
}
// the same with A resident in shared memory: planes of [box][128 rows][128 B]
template <int kD>
__device__ __forceinline__ void issue_cols_ss(uint32_t d, const UmmaDesc& a, uint32_t b_lo, uint32_t b_hi) {
  constexpr uint32_t idesc = umma_idesc(true, false, false, kBM, kBN);
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    const uint32_t at = a.lo + plane_of(kPlanesA, t) * umma_off(kBM * kD * 2), bt = b_lo + plane_of(kPlanesB, t) * umma_off(TileCfg<kD>::kPlane);
#pragma unroll
    for (int kk = 0; kk < kD / 16; ++kk)
      umma_ss_elect(d, at + umma_off((kk >> 2) * (kBM * 128) + (kk & 3) * 32), a.hi,
              bt + umma_off((kk >> 2) * kBoxBytes + (kk & 3) * 32), b_hi, idesc, kk > 0 || t > 0);
  }
}
// d[128 x kD] = A[128 x 64] (three planes in TMEM) * streamed tile[64 x kD]
template <int kD>
__device__ __forceinline__ void issue_dim(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t b_hi) {
  constexpr uint32_t idesc = umma_idesc(true, false, true, kBM, kD);
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    const uint32_t at = a + plane_of(kPlanesA, t) * 32, bt = b_lo + plane_of(kPlanesB, t) * umma_off(TileCfg<kD>::kPlane);
#pragma unroll
    for (int kk = 0; kk < kBN / 16; ++kk) umma_ts_elect(d, at + kk * 8, bt + umma_off(kk * 2048), b_hi, idesc, kk > 0 || t > 0);
  }
}

// The FMA forms (fma_rows_*), for CTAs whose results are not finite, by the math warps: a row is four neighbouring lanes,
// which deal the 16-byte pieces of the head dimension among them; a lane has pieces of two rows 64 apart, so that what it
// reads from shared memory, which bounds this, serves both.  The other sequence comes in tiles of 64 rows, in two
// buffers where the ring was.  B200, us, a NaN in V of every head, FMA kernels / these (with the tensor-core pass ahead
// of them) / a warp a row without staging: B4 H12 S1024 D64 causal forward 187 / 488 / 6349, backward 605 / 1338 / 12260;
// B2 Hq16 Hkv4 S1024 D128 forward 512 / 1083 / 10377; B1 H4 S4096 D64 causal (128 CTAs against 512) 264 / 1158 / 17704.
// The backward's are functions that are called, with nothing handed over but the block: inlined, two rows a lane in dK/dV
// too, they cost calls of finite values 2-3 % (B4 H12 S1024 155.5 against 154; the forward's costs nothing inlined).
constexpr int kLaneRows = 2;
// all math warps, with a bounded wait
struct RowSync {
  uint64_t* bar;
  volatile uint32_t* abort_flag;
  uint32_t* status;
  long long budget;
  uint32_t phase = 0;
  __device__ __forceinline__ bool operator()() {
    mbar_arrive_warp(bar);
    const bool ok = mbar_wait_warp(bar, phase, abort_flag, status, 0xf00, budget);
    phase ^= 1;
    return ok;
  }
};
// (its barrier is the last one of every kernel here)
template <class Cfg>
__device__ __forceinline__ RowSync row_sync(uint8_t* smem, uint32_t* status, long long budget) {
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kOffBars);
  return RowSync{bars + Cfg::kNumBars - 1, reinterpret_cast<uint32_t*>(bars + Cfg::kNumBars) + 1, status, budget};
}
// rows s0 + [0, 64) of a tensor to [row][kD]; zeros past the end
template <int kD>
__device__ __forceinline__ void stage_rows(float* dst, const View4& t, int b, int h, int s0, int rows) {
#pragma unroll
  for (int it = 0; it < kBN * kD / 4 / 256; ++it) {
    const int idx = static_cast<int>(threadIdx.x) + it * 256, r = idx / (kD / 4), c = idx % (kD / 4);
    const bool inside = s0 + r < rows;
    cp_async16(dst + r * kD + c * 4, row_ptr(t, b, h, inside ? s0 + r : 0) + c * 4, inside);
  }
}
// this lane's pieces of a row
template <int kD>
__device__ __forceinline__ void load_part(float2 (&x)[kD / 8], const float* row, int part) {
#pragma unroll
  for (int i = 0; i < kD / 16; ++i) {
    const float4 v = reinterpret_cast<const float4*>(row)[4 * i + part];
    x[2 * i] = make_float2(v.x, v.y);
    x[2 * i + 1] = make_float2(v.z, v.w);
  }
}
template <int kD>
__device__ __forceinline__ void store_part(float* row, int part, const float2 (&x)[kD / 8], float mul) {
#pragma unroll
  for (int i = 0; i < kD / 16; ++i)
    reinterpret_cast<float4*>(row)[4 * i + part] =
        make_float4(x[2 * i].x * mul, x[2 * i].y * mul, x[2 * i + 1].x * mul, x[2 * i + 1].y * mul);
}
// the products of a lane's rows with a streamed one, whole in all four lanes
template <int kD, int kN>
__device__ __forceinline__ void dot_parts(float (&s)[kN], const float2 (&x)[kN][kD / 8], const float* row, int part) {
  float2 a[kN], b[kN];
#pragma unroll
  for (int j = 0; j < kN; ++j) a[j] = b[j] = make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < kD / 16; ++i) {
    const float4 v = reinterpret_cast<const float4*>(row)[4 * i + part];
#pragma unroll
    for (int j = 0; j < kN; ++j) {
      a[j] = __ffma2_rn(x[j][2 * i], make_float2(v.x, v.y), a[j]);
      b[j] = __ffma2_rn(x[j][2 * i + 1], make_float2(v.z, v.w), b[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < kN; ++j) {
    s[j] = (a[j].x + a[j].y) + (b[j].x + b[j].y);
    s[j] += __shfl_xor_sync(0xffffffffu, s[j], 1);
    s[j] += __shfl_xor_sync(0xffffffffu, s[j], 2);
  }
}
// acc[j] += w[j] * the streamed row, for the rows that see it (`all`: every one).  A row that does not is left out: zero
// times what is not finite is not zero.
template <int kD, int kN>
__device__ __forceinline__ void add_parts(float2 (&acc)[kN][kD / 8], const float (&w)[kN], bool all, const bool (&sees)[kN],
                                          const float* row, int part) {
#pragma unroll
  for (int i = 0; i < kD / 16; ++i) {
    const float4 v = reinterpret_cast<const float4*>(row)[4 * i + part];
#pragma unroll
    for (int j = 0; j < kN; ++j) {
      const float2 w2 = make_float2(w[j], w[j]);
      const float2 lo = __ffma2_rn(w2, make_float2(v.x, v.y), acc[j][2 * i]), hi = __ffma2_rn(w2, make_float2(v.z, v.w), acc[j][2 * i + 1]);
      if (all || sees[j]) {
        acc[j][2 * i] = lo;
        acc[j][2 * i + 1] = hi;
      }
    }
  }
}

// Block index -> (row tile, head), the longest causal rows first over all heads
__device__ __forceinline__ void tile_and_head(int block, int tiles, int heads, bool latest_first, int* tile, int* bh) {
  const int t = block / heads;
  *bh = block - t * heads;
  *tile = latest_first ? tiles - 1 - t : t;
}

// ------------------------------------------------------------------------------------------
// forward.  TMEM columns: Q planes | S | P planes | the tile's P V.
// Order on the tensor pipe: S(0), S(1), then P V(j), S(j+2): S(j+2) and P V(j) run under the softmax of
// tile j + 1.
// ------------------------------------------------------------------------------------------
template <int kD>
struct FwdF32Cfg {
  using Tile = TileCfg<kD>;
  static constexpr int kSlots = kD == 64 ? 8 : 4;
  static constexpr int kOffX = kSlots * Tile::kBytes;         // [parity][half][row] maxima
  static constexpr int kOffBars = kOffX + 2 * 2 * kBM * 4;
  static constexpr int kNumBars = 2 * kSlots + 11;
  static constexpr int kSmemBytes = kOffBars + kNumBars * 8 + 16;
  static constexpr int kTmemQ = 0, kTmemS = 192, kTmemP = 256, kTmemO = 384;
};

template <int kD, bool kDropout>
__device__ __forceinline__ bool fma_rows_fwd(const FwdParams& p, int b, int h, int hk, int m0, int warp, int lane, uint8_t* smem, RowSync sync) {
  constexpr int kKeys = kD == 64 ? 4 : 2, kTile = kBN * kD;   // keys a step
  float* buf = reinterpret_cast<float*>(smem);   // [tile & 1][K, V][64][kD]
  const int part = lane & 3, bh = b * p.Hq + h;
  int q_row[kLaneRows], last[kLaneRows];
#pragma unroll
  for (int j = 0; j < kLaneRows; ++j) {
    q_row[j] = min(m0 + j * 64 + warp * 8 + (lane >> 2), p.Sq - 1);   // (rows past the end do the last one's work)
    last[j] = p.causal ? min(q_row[j] + p.causal_off, p.Sk - 1) : p.Sk - 1;
  }
  const int warp_first = __reduce_min_sync(0xffffffffu, last[0]), warp_last = __reduce_max_sync(0xffffffffu, last[1]);
  const int n_end = p.causal ? min(p.Sk, min(m0 + kBM, p.Sq) + p.causal_off) : p.Sk;
  const int tiles = (max(n_end, 0) + kBN - 1) / kBN;
  auto stage = [&](int t) {
    stage_rows<kD>(buf + (t & 1) * 2 * kTile, p.k, b, hk, t * kBN, p.Sk);
    stage_rows<kD>(buf + (t & 1) * 2 * kTile + kTile, p.v, b, hk, t * kBN, p.Sk);
    cp_commit();
  };
  float2 q[kLaneRows][kD / 8], o[kLaneRows][kD / 8];
  float m[kLaneRows], l[kLaneRows];
#pragma unroll
  for (int j = 0; j < kLaneRows; ++j) {
    load_part<kD>(q[j], row_ptr(p.q, b, h, q_row[j]), part);
#pragma unroll
    for (int i = 0; i < kD / 8; ++i) o[j][i] = make_float2(0.f, 0.f);
    m[j] = -INFINITY;
    l[j] = 0.f;
  }
  if (tiles > 0) stage(0);
#pragma unroll 1
  for (int t = 0; t < tiles; ++t) {
    cp_wait<0>();
    if (!sync()) return false;   // the tile is here, and everyone is done with the one before
    if (t + 1 < tiles) stage(t + 1);
    const float* kt = buf + (t & 1) * 2 * kTile;
    uint32_t keep[kLaneRows];
#pragma unroll 1
    for (int c = 0; c < kBN && t * kBN + c <= warp_last; c += kKeys) {
      const int k = t * kBN + c;
      if (kDropout && c % 16 == 0) {
#pragma unroll
        for (int j = 0; j < kLaneRows; ++j) keep[j] = dropout_bits16(p.drop, bh, q_row[j], k >> 4);
      }
      const bool all_see = k + kKeys - 1 <= warp_first;
      float s[kKeys][kLaneRows];
#pragma unroll
      for (int u = 0; u < kKeys; ++u) dot_parts<kD>(s[u], q, kt + (c + u) * kD, part);
#pragma unroll
      for (int j = 0; j < kLaneRows; ++j) {
        float m_new = m[j];
#pragma unroll
        for (int u = 0; u < kKeys; ++u) {
          if (!all_see && k + u > last[j]) s[u][j] = -INFINITY;
          m_new = fmaxf(m_new, s[u][j]);
        }
        if (m_new == -INFINITY) m_new = 0.f;
        const float corr = exp2f((m[j] - m_new) * p.scale_log2);
        m[j] = m_new;
        l[j] *= corr;
#pragma unroll
        for (int i = 0; i < kD / 8; ++i) o[j][i] = __fmul2_rn(o[j][i], make_float2(corr, corr));
#pragma unroll
        for (int u = 0; u < kKeys; ++u) {
          s[u][j] = exp2f((s[u][j] - m_new) * p.scale_log2);
          l[j] += s[u][j];
          if (kDropout && !((keep[j] >> ((c + u) & 15)) & 1u)) s[u][j] = 0.f;
        }
      }
#pragma unroll
      for (int u = 0; u < kKeys; ++u) {
        const bool sees[kLaneRows] = {k + u <= last[0], k + u <= last[1]};
        add_parts<kD>(o, s[u], all_see, sees, kt + kTile + (c + u) * kD, part);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < kLaneRows; ++j) {
    if (m0 + j * 64 + warp * 8 + (lane >> 2) >= p.Sq) continue;
    const float inv = l[j] > 0.f ? (kDropout ? p.drop.inv_keep : 1.f) / l[j] : 0.f;
    store_part<kD>(const_cast<float*>(row_ptr(p.out, b, h, q_row[j])), part, o[j], inv);
    if (part == 0) p.lse[static_cast<int64_t>(bh) * p.Sq + q_row[j]] = l[j] > 0.f ? m[j] * p.scale + logf(l[j]) : -INFINITY;
  }
  return true;
}

template <int kD, bool kDropout>
__global__ void __launch_bounds__(kThreads, 1) fwd_fp32_kernel(const __grid_constant__ FwdParams p) {
  using Cfg = FwdF32Cfg<kD>;
  using Tile = TileCfg<kD>;
  extern __shared__ __align__(1024) uint8_t smem[];
  float* sX = reinterpret_cast<float*>(smem + Cfg::kOffX);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kOffBars);
  uint64_t* full = bars;                     // [kSlots] a tile's planes are in shared memory (4 converter warps)
  uint64_t* empty = full + Cfg::kSlots;      // [kSlots]
  uint64_t* q_full = empty + Cfg::kSlots;    // Q planes in TMEM (8 math warps)
  uint64_t* s_full = q_full + 1;             // S ready
  uint64_t* s_free = s_full + 1;             // S read into registers (8)
  uint64_t* p_full = s_free + 1;             // P planes written, the last tile's P V read (8)
  uint64_t* pv_full = p_full + 1;            // P V ready, P planes consumed
  uint64_t* xchg = pv_full + 1;              // [4] the two warps of a row have written their half's maximum
  uint64_t* done = xchg + 4;                 // every math warp knows whether its results are finite (8)
  uint64_t* rows_done = done + 1;            // RowSync's (8)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + Cfg::kNumBars);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  volatile uint32_t* not_finite = tmem_slot + 2;

  const int warp = warp_index(), lane = threadIdx.x & 31;
  int tile, bh;
  tile_and_head(static_cast<int>(blockIdx.x), (p.Sq + kBM - 1) / kBM, p.B * p.Hq, p.causal, &tile, &bh);
  const int m0 = tile * kBM;
  const int b = bh / p.Hq, h = bh - b * p.Hq, hk = h / (p.Hq / p.Hkv);
  // key tiles: query row i sees key column j iff j <= i + causal_off; a row tile that sees no key runs one
  // masked step that gives zeros and -inf
  int n = (p.Sk + kBN - 1) / kBN;
  if (p.causal) {
    const int last = min(m0 + kBM - 1, p.Sq - 1) + p.causal_off;
    n = last < 0 ? 1 : min(n, last / kBN + 1);
  }

  if (status_is_set(p.status)) return;
  if ((smem_u32(smem) & 1023u) != 0u) {
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, kStatusOk, 0x414c0002u);
    return;
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < Cfg::kSlots; ++i) {
      mbar_init(&full[i], kConvWarps);
      mbar_init(&empty[i], 1);
    }
    mbar_init(q_full, kMathWarps);
    mbar_init(s_full, 1);
    mbar_init(s_free, kMathWarps);
    mbar_init(p_full, kMathWarps);
    mbar_init(pv_full, 1);
    for (int i = 0; i < 4; ++i) mbar_init(&xchg[i], 2);
    mbar_init(done, kMathWarps);
    mbar_init(rows_done, kMathWarps);
    *abort_flag = 0;
    *not_finite = 0;
    fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  if (warp < kMathWarps) {
    // =========================== math warps ===========================
    reg_alloc<kRegMath>();
    const int half = warp >> 2, r = (warp & 3) * 32 + lane, q_row = m0 + r;
    const uint32_t tm = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const float c = p.scale_log2;
    const float2 c2 = make_float2(c, c);
    {
      row_to_tmem<kD>(tm + Cfg::kTmemQ, p.q, b, h, q_row, p.Sq, half, kLift<kD>);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive_warp(q_full);
    }
    float o[kD / 2];   // this half of the head dim, relative to the row maximum as of the tile before
#pragma unroll
    for (int i = 0; i < kD / 2; ++i) o[i] = 0.f;
    float m = -INFINITY, sc = 0.f;   // row maximum, what the last tile scaled the sums by
    float2 l8[4];                    // this half's row sum, in eight parts: a sum of long rows rounds once per tile
#pragma unroll
    for (int i = 0; i < 4; ++i) l8[i] = make_float2(0.f, 0.f);
    for (int j = 0; j < n; ++j) {
      uint32_t keep = 0xffffffffu;
      if constexpr (kDropout) {
        const int blk = (j * kBN + half * 32) >> 4;
        keep = dropout_bits16(p.drop, bh, q_row, blk) | (dropout_bits16(p.drop, bh, q_row, blk + 1) << 16);
      }
      B200FA_WAIT(s_full, j & 1, 0xc00);
      tc_fence_after();
      float s[32];
      tmem_ld32(tm + Cfg::kTmemS + half * 32, reinterpret_cast<uint32_t*>(s));
      tmem_wait_ld();
      tc_fence_before();
      mbar_arrive_warp(s_free);
      const int col0 = j * kBN + half * 32;
      if ((p.causal && (j + 1) * kBN - 1 > m0 + p.causal_off) || (j + 1) * kBN > p.Sk) {
        const int last = p.causal ? min(q_row + p.causal_off, p.Sk - 1) : p.Sk - 1;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          if (col0 + i > last) s[i] = -INFINITY;
        }
      }
      float mx[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
      for (int i = 4; i < 32; ++i) mx[i & 3] = fmaxf(mx[i & 3], s[i]);
      const float mine = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      float* x = sX + (j & 1) * 2 * kBM + r;
      x[half * kBM] = mine;
      mbar_arrive_warp(&xchg[warp & 3]);
      B200FA_WAIT(&xchg[warp & 3], j & 1, 0xc10);
      float m_new = fmaxf(m, fmaxf(mine, x[(half ^ 1) * kBM]));
      if (m_new == -INFINITY) m_new = 0.f;
      const float sc_new = ex2_approx((m - m_new) * c);
      m = m_new;
      const float2 nm2 = make_float2(-m, -m);
#pragma unroll
      for (int i = 0; i < 4; ++i) l8[i] = __fmul2_rn(l8[i], make_float2(sc_new, sc_new));
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float2 a = __fmul2_rn(__fadd2_rn(make_float2(s[2 * i], s[2 * i + 1]), nm2), c2);
        const float2 pv = make_float2(ex2_approx(a.x), ex2_approx(a.y));
        l8[i & 3] = __fadd2_rn(l8[i & 3], pv);   // the row sum keeps every probability; only what multiplies V is dropped
        s[2 * i] = kDropout && !((keep >> (2 * i)) & 1u) ? 0.f : pv.x;
        s[2 * i + 1] = kDropout && !((keep >> (2 * i)) & 2u) ? 0.f : pv.y;
      }
      if (j > 0) {
        B200FA_WAIT(pv_full, (j - 1) & 1, 0xc20);
        tc_fence_after();
        add_part<kD / 64>(o, tm + Cfg::kTmemO + half * (kD / 2), sc);
      }
      sc = sc_new;
      values_to_tmem(tm + Cfg::kTmemP, s, half);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive_warp(p_full);
    }
    float l;
    {
      const float2 a = __fadd2_rn(__fadd2_rn(l8[0], l8[1]), __fadd2_rn(l8[2], l8[3]));
      l = a.x + a.y;
      float* x = sX + (n & 1) * 2 * kBM + r;
      x[half * kBM] = l;
      mbar_arrive_warp(&xchg[warp & 3]);
      B200FA_WAIT(&xchg[warp & 3], n & 1, 0xc11);
      l += x[(half ^ 1) * kBM];
    }
    B200FA_WAIT(pv_full, (n - 1) & 1, 0xc21);
    tc_fence_after();
    add_part<kD / 64>(o, tm + Cfg::kTmemO + half * (kD / 2), sc);
    // the row sum too: where dropout drops a key whose probability is NaN, only that knows of it
    if (q_row < p.Sq && (!all_finite(o) || !(l < INFINITY))) *not_finite = 1;
    mbar_arrive_warp(done);
    B200FA_WAIT(done, 0, 0xc30);
    if (*not_finite) {
      if (!fma_rows_fwd<kD, kDropout>(p, b, h, hk, m0, warp, lane, smem, RowSync{rows_done, abort_flag, p.status, p.wait_budget})) goto teardown;
    } else if (q_row < p.Sq) {
      const float inv = l > 0.f ? (kDropout ? p.drop.inv_keep : 1.f) / l : 0.f;
      float4* dst = reinterpret_cast<float4*>(const_cast<float*>(row_ptr(p.out, b, h, q_row)) + half * (kD / 2));
#pragma unroll
      for (int i = 0; i < kD / 8; ++i)
        dst[i] = make_float4(o[4 * i] * inv, o[4 * i + 1] * inv, o[4 * i + 2] * inv, o[4 * i + 3] * inv);
      if (half == 0)
        p.lse[(static_cast<int64_t>(b) * p.Hq + h) * p.Sq + q_row] = l > 0.f ? m * p.scale + logf(l) : -INFINITY;
    }
  } else if (warp < kConvWarp0 + kConvWarps) {
    // =========================== converters ===========================
    reg_dealloc<kRegConv>();
    // the tiles in the order the MMAs take them: K_0, K_1, V_0, K_2, V_1, ...
    const int tid = threadIdx.x - kConvWarp0 * 32;
    auto load = [&](float4 (&v)[8], int seq, int box) {
      const bool is_k = seq == 0 || ((seq & 1) && seq != 2 * n - 1);
      const int j = is_k ? (seq + 1) >> 1 : seq == 2 * n - 1 ? n - 1 : (seq >> 1) - 1;
      load_box(v, is_k ? p.k : p.v, b, hk, j * kBN, p.Sk, box * 64, tid);
    };
    // box i of the stream is split while the loads of box i + 1 are in flight (two sets of registers that
    // change places: a copy would wait for the loads)
    const int boxes = 2 * n * Tile::kBoxes;
    auto step = [&](int i, float4 (&now)[8], float4 (&next)[8]) -> bool {
      const int seq = i / Tile::kBoxes, box = i % Tile::kBoxes, slot = seq % Cfg::kSlots;
      if (i + 1 < boxes) load(next, (i + 1) / Tile::kBoxes, (i + 1) % Tile::kBoxes);
      if (box == 0 && seq >= Cfg::kSlots &&
          !mbar_wait(&empty[slot], (seq / Cfg::kSlots - 1) & 1, abort_flag, p.status, 0xc40, p.wait_budget)) return false;
      store_box(now, smem + slot * Tile::kBytes + box * kBoxBytes, Tile::kPlane, tid);
      if (box == Tile::kBoxes - 1) {
        fence_proxy_async_smem();
        mbar_arrive_warp(&full[slot]);
      }
      return true;
    };
    float4 v0[8], v1[8];
    load(v0, 0, 0);
    for (int i = 0; i < boxes; i += 2) {
      if (!step(i, v0, v1) || !step(i + 1, v1, v0)) goto teardown;
    }
  } else {
    reg_dealloc<kRegRest>();
    if (warp == kMmaWarp) {
      // =========================== MMA issuer ===========================
      const uint32_t tQ = tmem_base + Cfg::kTmemQ, tS = tmem_base + Cfg::kTmemS, tP = tmem_base + Cfg::kTmemP,
                     tO = tmem_base + Cfg::kTmemO;
      const UmmaDesc dK = umma_desc_split(smem_u32(smem), 16, 1024), dV = umma_desc_split(smem_u32(smem), kBoxBytes, 1024);
      constexpr uint32_t kSlotLo = umma_off(Tile::kBytes);
      B200FA_WAIT_WARP(q_full, 0, 0xc50);
      for (int j = -2; j < n; ++j) {
        if (j >= 0) {
          const int seq = j == n - 1 ? 2 * n - 1 : 2 * j + 2, slot = seq % Cfg::kSlots;
          B200FA_WAIT_WARP(&full[slot], (seq / Cfg::kSlots) & 1, 0xc51);
          B200FA_WAIT_WARP(p_full, j & 1, 0xc52);
          tc_fence_after();
          issue_dim<kD>(tO, tP, dV.lo + slot * kSlotLo, dV.hi);
          umma_commit_elect(pv_full);
          umma_commit_elect(&empty[slot]);
        }
        const int js = j + 2;   // the tile whose scores come next
        if (js < n) {
          const int seq = js == 0 ? 0 : 2 * js - 1, slot = seq % Cfg::kSlots;
          B200FA_WAIT_WARP(&full[slot], (seq / Cfg::kSlots) & 1, 0xc53);
          if (js > 0) { B200FA_WAIT_WARP(s_free, (js - 1) & 1, 0xc54); }
          tc_fence_after();
          issue_cols_ts<kD>(tS, tQ, dK.lo + slot * kSlotLo, dK.hi);
          umma_commit_elect(s_full);
          umma_commit_elect(&empty[slot]);
        }
      }
    }
  }

teardown:
  tc_fence_before();
  __syncthreads();
  settle_if_aborted(abort_flag);
  if (warp == kMmaWarp) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------------------------
// backward, dQ: resident query rows, K and V streamed.  TMEM columns: Q planes | dO planes | S | dP |
// dS planes | the tile's dS K.  Tensor pipe: S(0) dP(0), S(1) dP(1), then dQ(j), S(j+2) dP(j+2).
// ------------------------------------------------------------------------------------------
template <int kD>
struct DqF32Cfg {
  using Tile = TileCfg<kD>;
  static constexpr int kSlots = 8;
  static constexpr int kOffBars = kSlots * Tile::kBytes;
  static constexpr int kNumBars = 2 * kSlots + 7;
  static constexpr int kSmemBytes = kOffBars + kNumBars * 8 + 16;
  static constexpr int kTmemQ = 0, kTmemDO = 96, kTmemS = 192, kTmemDP = 256, kTmemDS = 320, kTmemDQ = 448;
};

template <int kD, bool kDropout>
__device__ __noinline__ bool fma_rows_dq(const BwdParams& p, int block, uint8_t* smem) {
  RowSync sync = row_sync<DqF32Cfg<kD>>(smem, p.status, p.wait_budget);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int tile, bh;
  tile_and_head(block, (p.S + kBM - 1) / kBM, p.B * p.Hq, p.causal, &tile, &bh);
  const int m0 = tile * kBM, b = bh / p.Hq, h = bh - b * p.Hq, hk = h / (p.Hq / p.Hkv);
  constexpr int kKeys = 2, kTile = kBN * kD;
  float* buf = reinterpret_cast<float*>(smem);   // [tile & 1][K, V][64][kD]
  const int part = lane & 3;
  int q_row[kLaneRows], last[kLaneRows];
#pragma unroll
  for (int j = 0; j < kLaneRows; ++j) {
    q_row[j] = min(m0 + j * 64 + warp * 8 + (lane >> 2), p.S - 1);   // (rows past the end do the last one's work)
    last[j] = p.causal ? min(q_row[j] + p.causal_off, p.Sk - 1) : p.Sk - 1;
  }
  const int warp_first = __reduce_min_sync(0xffffffffu, last[0]), warp_last = __reduce_max_sync(0xffffffffu, last[1]);
  const int n_end = p.causal ? min(p.Sk, min(m0 + kBM, p.S) + p.causal_off) : p.Sk;
  const int tiles = (max(n_end, 0) + kBN - 1) / kBN;
  auto stage = [&](int t) {
    stage_rows<kD>(buf + (t & 1) * 2 * kTile, p.k, b, hk, t * kBN, p.Sk);
    stage_rows<kD>(buf + (t & 1) * 2 * kTile + kTile, p.v, b, hk, t * kBN, p.Sk);
    cp_commit();
  };
  float2 q[kLaneRows][kD / 8], g[kLaneRows][kD / 8], dq[kLaneRows][kD / 8];
  float l2[kLaneRows], dps[kLaneRows];
#pragma unroll
  for (int j = 0; j < kLaneRows; ++j) {
    load_part<kD>(q[j], row_ptr(p.q, b, h, q_row[j]), part);
    load_part<kD>(g[j], row_ptr(p.dout, b, h, q_row[j]), part);
#pragma unroll
    for (int i = 0; i < kD / 8; ++i) dq[j][i] = make_float2(0.f, 0.f);
    const float lse = p.lse[static_cast<int64_t>(bh) * p.S + q_row[j]];
    l2[j] = lse != -INFINITY ? lse * kLog2e : INFINITY;
    dps[j] = __ldcg(p.dpsum + static_cast<int64_t>(bh) * p.Spad + q_row[j]);
  }
  if (tiles > 0) stage(0);
#pragma unroll 1
  for (int t = 0; t < tiles; ++t) {
    cp_wait<0>();
    if (!sync()) return false;   // the tile is here, and everyone is done with the one before
    if (t + 1 < tiles) stage(t + 1);
    const float* kt = buf + (t & 1) * 2 * kTile;
    uint32_t keep[kLaneRows];
#pragma unroll 1
    for (int c = 0; c < kBN && t * kBN + c <= warp_last; c += kKeys) {
      const int k = t * kBN + c;
      if (kDropout && c % 16 == 0) {
#pragma unroll
        for (int j = 0; j < kLaneRows; ++j) keep[j] = dropout_bits16(p.drop, bh, q_row[j], k >> 4);
      }
      const bool all_see = k + kKeys - 1 <= warp_first;
      float s[kKeys][kLaneRows], dp[kKeys][kLaneRows];
#pragma unroll
      for (int u = 0; u < kKeys; ++u) {
        dot_parts<kD>(s[u], q, kt + (c + u) * kD, part);
        dot_parts<kD>(dp[u], g, kt + kTile + (c + u) * kD, part);
#pragma unroll
        for (int j = 0; j < kLaneRows; ++j) {
          if (kDropout) dp[u][j] *= (keep[j] >> ((c + u) & 15)) & 1u ? p.drop.inv_keep : 0.f;
          s[u][j] = exp2f(s[u][j] * p.scale_log2 - l2[j]) * (dp[u][j] - dps[j]);
        }
      }
#pragma unroll
      for (int u = 0; u < kKeys; ++u) {
        const bool sees[kLaneRows] = {k + u <= last[0], k + u <= last[1]};
        add_parts<kD>(dq, s[u], all_see, sees, kt + (c + u) * kD, part);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < kLaneRows; ++j) {
    if (m0 + j * 64 + warp * 8 + (lane >> 2) < p.S) store_part<kD>(const_cast<float*>(row_ptr(p.dq, b, h, q_row[j])), part, dq[j], p.scale);
  }
  return true;
}

template <int kD, bool kDropout>
__device__ __forceinline__ void dq_block(const BwdParams& p, int block, uint8_t* smem) {
  using Cfg = DqF32Cfg<kD>;
  using Tile = TileCfg<kD>;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kOffBars);
  uint64_t* full = bars;                     // [kSlots] (4 converter warps)
  uint64_t* empty = full + Cfg::kSlots;      // [kSlots]
  uint64_t* q_full = empty + Cfg::kSlots;    // Q and dO planes in TMEM (8 math warps)
  uint64_t* s_full = q_full + 1;             // S and dP ready
  uint64_t* s_free = s_full + 1;             // S and dP read into registers (8)
  uint64_t* ds_full = s_free + 1;            // dS planes written, the last tile's dS K read (8)
  uint64_t* dq_full = ds_full + 1;           // dS K ready, dS planes consumed
  uint64_t* done = dq_full + 1;              // (8)
  uint64_t* rows_done = done + 1;            // RowSync's (8)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + Cfg::kNumBars);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  volatile uint32_t* not_finite = tmem_slot + 2;

  const int warp = warp_index(), lane = threadIdx.x & 31;
  int tile, bh;
  tile_and_head(block, (p.S + kBM - 1) / kBM, p.B * p.Hq, p.causal, &tile, &bh);
  const int m0 = tile * kBM;
  const int b = bh / p.Hq, h = bh - b * p.Hq, hk = h / (p.Hq / p.Hkv);
  int n = (p.Sk + kBN - 1) / kBN;   // key tiles (none: dQ is zero)
  if (p.causal) {
    const int last = min(m0 + kBM - 1, p.S - 1) + p.causal_off;
    n = last < 0 ? 0 : min(n, last / kBN + 1);
  }

  if (threadIdx.x == 0) {
    for (int i = 0; i < Cfg::kSlots; ++i) {
      mbar_init(&full[i], kConvWarps);
      mbar_init(&empty[i], 1);
    }
    mbar_init(q_full, kMathWarps);
    mbar_init(s_full, 1);
    mbar_init(s_free, kMathWarps);
    mbar_init(ds_full, kMathWarps);
    mbar_init(dq_full, 1);
    mbar_init(done, kMathWarps);
    mbar_init(rows_done, kMathWarps);
    *abort_flag = 0;
    *not_finite = 0;
    fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  if (warp < kMathWarps) {
    // =========================== math warps ===========================
    reg_alloc<kRegMath>();
    const int half = warp >> 2, r = (warp & 3) * 32 + lane, q_row = m0 + r;
    const uint32_t tm = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const float c = p.scale_log2;
    const float2 c2 = make_float2(c, c);
    float nl2 = -INFINITY, ndps = 0.f;   // minus the row's statistics; rows past the end, and rows that saw no key: P = 0
    {
      row_to_tmem<kD>(tm + Cfg::kTmemQ, p.q, b, h, q_row, p.S, half, kLift<kD>);
      row_to_tmem<kD>(tm + Cfg::kTmemDO, p.dout, b, h, q_row, p.S, half, 0.f);
      if (q_row < p.S) {
        const float lse = p.lse[static_cast<int64_t>(bh) * p.S + q_row];
        if (lse != -INFINITY) nl2 = -(lse * kLog2e);
        ndps = -__ldcg(p.dpsum + static_cast<int64_t>(bh) * p.Spad + q_row);
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive_warp(q_full);
    }
    const float2 nl22 = make_float2(nl2, nl2), nd2 = make_float2(ndps, ndps);
    float dq[kD / 2];
#pragma unroll
    for (int i = 0; i < kD / 2; ++i) dq[i] = 0.f;
    for (int j = 0; j < n; ++j) {
      uint32_t keep = 0xffffffffu;
      if constexpr (kDropout) {
        const int blk = (j * kBN + half * 32) >> 4;
        keep = dropout_bits16(p.drop, bh, q_row, blk) | (dropout_bits16(p.drop, bh, q_row, blk + 1) << 16);
      }
      B200FA_WAIT(s_full, j & 1, 0xd00);
      tc_fence_after();
      float s[32], dp[32];
      tmem_ld32(tm + Cfg::kTmemS + half * 32, reinterpret_cast<uint32_t*>(s));
      tmem_ld32(tm + Cfg::kTmemDP + half * 32, reinterpret_cast<uint32_t*>(dp));
      tmem_wait_ld();
      tc_fence_before();
      mbar_arrive_warp(s_free);
      const int col0 = j * kBN + half * 32;
      const bool need_mask = (p.causal && (j + 1) * kBN - 1 > m0 + p.causal_off) || (j + 1) * kBN > p.Sk;
      const int last = p.causal ? min(q_row + p.causal_off, p.Sk - 1) : p.Sk - 1;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float2 a = __ffma2_rn(make_float2(s[2 * i], s[2 * i + 1]), c2, nl22);
        float2 pv = make_float2(ex2_approx(a.x), ex2_approx(a.y));
        if (need_mask) {
          if (col0 + 2 * i > last) pv.x = 0.f;
          if (col0 + 2 * i + 1 > last) pv.y = 0.f;
        }
        float2 g = make_float2(dp[2 * i], dp[2 * i + 1]);
        if constexpr (kDropout) {
          g.x = (keep >> (2 * i)) & 1u ? g.x * p.drop.inv_keep : 0.f;
          g.y = (keep >> (2 * i)) & 2u ? g.y * p.drop.inv_keep : 0.f;
        }
        const float2 ds = __fmul2_rn(pv, __fadd2_rn(g, nd2));
        s[2 * i] = ds.x;
        s[2 * i + 1] = ds.y;
      }
      if (j > 0) {
        B200FA_WAIT(dq_full, (j - 1) & 1, 0xd20);
        tc_fence_after();
        add_part<kD / 64>(dq, tm + Cfg::kTmemDQ + half * (kD / 2), 1.f);
      }
      values_to_tmem(tm + Cfg::kTmemDS, s, half);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive_warp(ds_full);
    }
    if (n > 0) {
      B200FA_WAIT(dq_full, (n - 1) & 1, 0xd21);
      tc_fence_after();
      add_part<kD / 64>(dq, tm + Cfg::kTmemDQ + half * (kD / 2), 1.f);
    }
    if (q_row < p.S && !all_finite(dq)) *not_finite = 1;
    mbar_arrive_warp(done);
    B200FA_WAIT(done, 0, 0xd30);
    if (*not_finite) {
      if (!fma_rows_dq<kD, kDropout>(p, block, smem)) goto teardown;
    } else if (q_row < p.S) {
      float4* dst = reinterpret_cast<float4*>(const_cast<float*>(row_ptr(p.dq, b, h, q_row)) + half * (kD / 2));
#pragma unroll
      for (int i = 0; i < kD / 8; ++i)
        dst[i] = make_float4(dq[4 * i] * p.scale, dq[4 * i + 1] * p.scale, dq[4 * i + 2] * p.scale, dq[4 * i + 3] * p.scale);
    }
  } else if (warp < kConvWarp0 + kConvWarps) {
    // =========================== converters: K_0, V_0, K_1, V_1, ... ===========================
    reg_dealloc<kRegConv>();
    const int tid = threadIdx.x - kConvWarp0 * 32;
    auto step = [&](int seq, float4 (&now)[8], float4 (&next)[8]) -> bool {
      const int slot = seq % Cfg::kSlots;
      if (seq + 1 < 2 * n) load_box(next, (seq & 1) ? p.k : p.v, b, hk, ((seq + 1) >> 1) * kBN, p.Sk, 0, tid);
      if (seq >= Cfg::kSlots &&
          !mbar_wait(&empty[slot], (seq / Cfg::kSlots - 1) & 1, abort_flag, p.status, 0xd40, p.wait_budget)) return false;
      store_box(now, smem + slot * Tile::kBytes, Tile::kPlane, tid);
      fence_proxy_async_smem();
      mbar_arrive_warp(&full[slot]);
      return true;
    };
    float4 v0[8], v1[8];
    if (n > 0) load_box(v0, p.k, b, hk, 0, p.Sk, 0, tid);
    for (int seq = 0; seq < 2 * n; seq += 2) {
      if (!step(seq, v0, v1) || !step(seq + 1, v1, v0)) goto teardown;
    }
  } else {
    reg_dealloc<kRegRest>();
    if (warp == kMmaWarp) {
      // =========================== MMA issuer ===========================
      const uint32_t tQ = tmem_base + Cfg::kTmemQ, tDO = tmem_base + Cfg::kTmemDO, tS = tmem_base + Cfg::kTmemS,
                     tDP = tmem_base + Cfg::kTmemDP, tDS = tmem_base + Cfg::kTmemDS, tDQ = tmem_base + Cfg::kTmemDQ;
      const UmmaDesc dCols = umma_desc_split(smem_u32(smem), 16, 1024), dDim = umma_desc_split(smem_u32(smem), kBoxBytes, 1024);
      constexpr uint32_t kSlotLo = umma_off(Tile::kBytes);
      if (n > 0) { B200FA_WAIT_WARP(q_full, 0, 0xd50); }
      for (int j = -2; j < n; ++j) {
        if (j >= 0) {
          const int slot = (2 * j) % Cfg::kSlots;   // K_j has been waited for
          B200FA_WAIT_WARP(ds_full, j & 1, 0xd52);
          tc_fence_after();
          issue_dim<kD>(tDQ, tDS, dDim.lo + slot * kSlotLo, dDim.hi);
          umma_commit_elect(dq_full);
          umma_commit_elect(&empty[slot]);
        }
        const int js = j + 2;
        if (js < n) {
          const int seq = 2 * js, slot = seq % Cfg::kSlots;   // K_js, V_js right behind it
          const uint32_t parity = (seq / Cfg::kSlots) & 1;
          B200FA_WAIT_WARP(&full[slot], parity, 0xd53);
          if (js > 0) { B200FA_WAIT_WARP(s_free, (js - 1) & 1, 0xd54); }
          tc_fence_after();
          issue_cols_ts<kD>(tS, tQ, dCols.lo + slot * kSlotLo, dCols.hi);
          B200FA_WAIT_WARP(&full[slot + 1], parity, 0xd55);
          tc_fence_after();
          issue_cols_ts<kD>(tDP, tDO, dCols.lo + (slot + 1) * kSlotLo, dCols.hi);
          umma_commit_elect(s_full);
          umma_commit_elect(&empty[slot + 1]);
        }
      }
    }
  }

teardown:
  tc_fence_before();
  __syncthreads();
  settle_if_aborted(abort_flag);
  if (warp == kMmaWarp) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------------------------
// backward, dK and dV: resident key rows (K and V planes in shared memory), Q and dO streamed for
// every query head of the group.  TMEM columns: S^T | dP^T | P^T planes | dS^T planes | the tile's
// P^T dO | the tile's dS^T Q.
// ------------------------------------------------------------------------------------------
template <int kD>
struct DkdvF32Cfg {
  using Tile = TileCfg<kD>;
  static constexpr int kSlots = 5;
  static constexpr int kResPlane = kBM * kD * 2;                 // one plane of K or V
  static constexpr int kOffK = 0, kOffV = 3 * kResPlane, kOffStream = 6 * kResPlane;
  static constexpr int kStats = 4;                               // tiles whose statistics are kept
  static constexpr int kOffStat = kOffStream + kSlots * Tile::kBytes;   // [tile & 3][lse2 | dpsum][64], both negated
  static constexpr int kOffBars = kOffStat + kStats * 2 * kBN * 4;
  static constexpr int kNumBars = 2 * kSlots + 7;
  static constexpr int kSmemBytes = kOffBars + kNumBars * 8 + 16;
  static constexpr int kTmemS = 0, kTmemDP = 64, kTmemP = 128, kTmemDS = 224, kTmemDV = 320, kTmemDK = 384;
};

template <int kD, bool kDropout>
__device__ __noinline__ bool fma_rows_dkdv(const BwdParams& p, int block, uint8_t* smem) {
  RowSync sync = row_sync<DkdvF32Cfg<kD>>(smem, p.status, p.wait_budget);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int tile, bhk;
  tile_and_head(block, (p.Sk + kBM - 1) / kBM, p.B * p.Hkv, false, &tile, &bhk);
  const int n0 = tile * kBM, b = bhk / p.Hkv, hk = bhk - b * p.Hkv;
  constexpr int kN = 1, kTile = kBN * kD;   // (two rows a lane do not fit: 128 registers of operands and sums)
  float* buf = reinterpret_cast<float*>(smem);   // [tile & 1][Q, dO][64][kD]
  const int part = lane & 3, group = p.Hq / p.Hkv;
#pragma unroll 1
  for (int row0 = n0; row0 < min(n0 + kBM, p.Sk); row0 += 64) {
    int key[kN], first[kN];   // first query row that sees the key
#pragma unroll
    for (int j = 0; j < kN; ++j) {
      key[j] = min(row0 + j * 64 + warp * 8 + (lane >> 2), p.Sk - 1);
      first[j] = p.causal ? max(0, key[j] - p.causal_off) : 0;
    }
    const int warp_first = __reduce_min_sync(0xffffffffu, first[0]), warp_last = __reduce_max_sync(0xffffffffu, first[kN - 1]);
    const int m_begin = p.causal ? max(0, row0 - p.causal_off) / kBN * kBN : 0;
    const int per_head = max(0, (p.S - m_begin + kBN - 1) / kBN), tiles = group * per_head;
    auto stage = [&](int t) {
      const int h = hk * group + t / per_head, q0 = m_begin + t % per_head * kBN;
      stage_rows<kD>(buf + (t & 1) * 2 * kTile, p.q, b, h, q0, p.S);
      stage_rows<kD>(buf + (t & 1) * 2 * kTile + kTile, p.dout, b, h, q0, p.S);
      cp_commit();
    };
    float2 k[kN][kD / 8], v[kN][kD / 8], dk[kN][kD / 8], dv[kN][kD / 8];
#pragma unroll
    for (int j = 0; j < kN; ++j) {
      load_part<kD>(k[j], row_ptr(p.k, b, hk, key[j]), part);
      load_part<kD>(v[j], row_ptr(p.v, b, hk, key[j]), part);
#pragma unroll
      for (int i = 0; i < kD / 8; ++i) dk[j][i] = dv[j][i] = make_float2(0.f, 0.f);
    }
    if (tiles > 0) stage(0);
#pragma unroll 1
    for (int t = 0; t < tiles; ++t) {
      cp_wait<0>();
      if (!sync()) return false;
      if (t + 1 < tiles) stage(t + 1);
      const float* qt = buf + (t & 1) * 2 * kTile;
      const int bh = b * p.Hq + hk * group + t / per_head, q0 = m_begin + t % per_head * kBN;
#pragma unroll 1
      for (int c0 = 0; c0 < kBN && q0 + c0 < p.S; c0 += 32) {
        // lane L has the statistics of query row L of these 32, and its keep bits against the 16 keys that hold this warp's
        const int mine = min(q0 + c0 + lane, p.S - 1);
        const float lse = p.lse[static_cast<int64_t>(bh) * p.S + mine], my_dps = __ldcg(p.dpsum + static_cast<int64_t>(bh) * p.Spad + mine);
        const float my_l2 = lse != -INFINITY ? lse * kLog2e : INFINITY;
        uint32_t my_keep[kN];
        if constexpr (kDropout) {
#pragma unroll
          for (int j = 0; j < kN; ++j) my_keep[j] = dropout_bits16(p.drop, bh, mine, (row0 + j * 64 + warp * 8) >> 4);
        }
#pragma unroll 1
        for (int u = max(0, warp_first - q0 - c0); u < min(32, p.S - q0 - c0); ++u) {
          const float l2 = __shfl_sync(0xffffffffu, my_l2, u), dps = __shfl_sync(0xffffffffu, my_dps, u);
          const float* qr = qt + (c0 + u) * kD;
          float s[kN], dp[kN];
          dot_parts<kD>(s, k, qr, part);
          dot_parts<kD>(dp, v, qr + kTile, part);
#pragma unroll
          for (int j = 0; j < kN; ++j) {
            const float pv = exp2f(s[j] * p.scale_log2 - l2);
            float dm = 1.f;
            if constexpr (kDropout) dm = (__shfl_sync(0xffffffffu, my_keep[j], u) >> (key[j] & 15)) & 1u ? p.drop.inv_keep : 0.f;
            s[j] = pv * dm;
            dp[j] = pv * (dp[j] * dm - dps);
          }
          const int q_row = q0 + c0 + u;
          const bool sees[kN] = {q_row >= first[0]};
          add_parts<kD>(dv, s, q_row >= warp_last, sees, qr + kTile, part);
          add_parts<kD>(dk, dp, q_row >= warp_last, sees, qr, part);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < kN; ++j) {
      if (row0 + j * 64 + warp * 8 + (lane >> 2) >= p.Sk) continue;
      store_part<kD>(const_cast<float*>(row_ptr(p.dk, b, hk, key[j])), part, dk[j], p.scale);
      store_part<kD>(const_cast<float*>(row_ptr(p.dv, b, hk, key[j])), part, dv[j], 1.f);
    }
    if (!sync()) return false;   // the next pass writes the buffers
  }
  return true;
}

template <int kD, bool kDropout>
__device__ __forceinline__ void dkdv_block(const BwdParams& p, int block, uint8_t* smem) {
  using Cfg = DkdvF32Cfg<kD>;
  using Tile = TileCfg<kD>;
  float* sStat = reinterpret_cast<float*>(smem + Cfg::kOffStat);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kOffBars);
  uint64_t* full = bars;                     // [kSlots] (4 converter warps)
  uint64_t* empty = full + Cfg::kSlots;      // [kSlots]
  uint64_t* kv_full = empty + Cfg::kSlots;   // K and V planes in shared memory (8 math warps)
  uint64_t* s_full = kv_full + 1;            // S^T and dP^T ready
  uint64_t* s_free = s_full + 1;             // ... read into registers (8)
  uint64_t* ds_full = s_free + 1;            // P^T and dS^T planes written, the last tile's products read (8)
  uint64_t* acc_full = ds_full + 1;          // P^T dO and dS^T Q ready, the planes consumed
  uint64_t* done = acc_full + 1;             // (8)
  uint64_t* rows_done = done + 1;            // RowSync's (8)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + Cfg::kNumBars);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  volatile uint32_t* not_finite = tmem_slot + 2;

  const int warp = warp_index(), lane = threadIdx.x & 31;
  int tile, bhk;
  tile_and_head(block, (p.Sk + kBM - 1) / kBM, p.B * p.Hkv, false, &tile, &bhk);
  const int n0 = tile * kBM;
  const int b = bhk / p.Hkv, hk = bhk - b * p.Hkv, group = p.Hq / p.Hkv;
  const int m_begin = p.causal ? max(0, n0 - p.causal_off) / kBN * kBN : 0;   // first tile with a query that sees a key
  const int per_head = max(0, (p.S - m_begin + kBN - 1) / kBN);
  const int n = group * per_head;

  if (threadIdx.x == 0) {
    for (int i = 0; i < Cfg::kSlots; ++i) {
      mbar_init(&full[i], kConvWarps);
      mbar_init(&empty[i], 1);
    }
    mbar_init(kv_full, kMathWarps);
    mbar_init(s_full, 1);
    mbar_init(s_free, kMathWarps);
    mbar_init(ds_full, kMathWarps);
    mbar_init(acc_full, 1);
    mbar_init(done, kMathWarps);
    mbar_init(rows_done, kMathWarps);
    *abort_flag = 0;
    *not_finite = 0;
    fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  if (warp < kMathWarps) {
    // =========================== math warps ===========================
    reg_alloc<kRegMath>();
    const int half = warp >> 2, r = (warp & 3) * 32 + lane;   // half of the query columns; key row
    const uint32_t tm = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const float c = p.scale_log2;
    const float2 c2 = make_float2(c, c);
    {
#pragma unroll
      for (int which = 0; which < 2; ++which) {
#pragma unroll
        for (int box = 0; box < Tile::kBoxes; ++box)
#pragma unroll
          for (int it = 0; it < kBM * 8 / 256; ++it) {
            const int idx = threadIdx.x + it * 256, row = idx >> 3, piece = idx & 7;
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
            if (n0 + row < p.Sk) {
              const float4* src = reinterpret_cast<const float4*>(row_ptr(which == 0 ? p.k : p.v, b, hk, n0 + row) + box * 64 + piece * 8);
              x = src[0];
              y = src[1];
            }
            store_piece(smem + (which == 0 ? Cfg::kOffK : Cfg::kOffV) + box * kBM * 128, Cfg::kResPlane, row, piece, x, y, which == 0 ? kLift<kD> : 0.f);
          }
      }
      fence_proxy_async_smem();
      mbar_arrive_warp(kv_full);
    }
    float dk[kD / 2], dv[kD / 2];
#pragma unroll
    for (int i = 0; i < kD / 2; ++i) dk[i] = dv[i] = 0.f;
    int h = hk * group, m0 = m_begin;   // of this tile
    for (int j = 0; j < n; ++j) {
      uint32_t keep = 0xffffffffu;
      if constexpr (kDropout) {
        // lane L draws the bits of query row L against this warp's 32 key rows, and the warp transposes them
        const int blk = (n0 + (warp & 3) * 32) >> 4, q_row = m0 + half * 32 + lane, bh = b * p.Hq + h;
        keep = warp_transpose_bits(dropout_bits16(p.drop, bh, q_row, blk) | (dropout_bits16(p.drop, bh, q_row, blk + 1) << 16));
      }
      const int slot = (2 * j) % Cfg::kSlots;
      // the statistics came with the Q tile
      B200FA_WAIT(&full[slot], (2 * j / Cfg::kSlots) & 1, 0xe01);
      B200FA_WAIT(s_full, j & 1, 0xe00);
      tc_fence_after();
      float s[32], dp[32];
      tmem_ld32(tm + Cfg::kTmemS + half * 32, reinterpret_cast<uint32_t*>(s));
      tmem_ld32(tm + Cfg::kTmemDP + half * 32, reinterpret_cast<uint32_t*>(dp));
      tmem_wait_ld();
      tc_fence_before();
      mbar_arrive_warp(s_free);
      const float4* nl2 = reinterpret_cast<const float4*>(sStat + (j % Cfg::kStats) * 2 * kBN + half * 32);
      const float4* ndps = nl2 + kBN / 4;
      const bool need_mask = p.causal && n0 + kBM - 1 > m0 + p.causal_off;
      const int first_q = n0 + r - p.causal_off - (m0 + half * 32);   // first of these 32 columns that sees this key
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 l4 = nl2[i], d4 = ndps[i];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int e = 4 * i + 2 * u;
          const float2 a = __ffma2_rn(make_float2(s[e], s[e + 1]), c2, u ? make_float2(l4.z, l4.w) : make_float2(l4.x, l4.y));
          float2 pv = make_float2(ex2_approx(a.x), ex2_approx(a.y));
          if (need_mask) {
            if (e < first_q) pv.x = 0.f;
            if (e + 1 < first_q) pv.y = 0.f;
          }
          float2 g = make_float2(dp[e], dp[e + 1]), pd = pv;
          if constexpr (kDropout) {
            const float k0 = (keep >> e) & 1u ? p.drop.inv_keep : 0.f, k1 = (keep >> e) & 2u ? p.drop.inv_keep : 0.f;
            g = make_float2(g.x * k0, g.y * k1);
            pd = make_float2(pv.x * k0, pv.y * k1);
          }
          const float2 ds = __fmul2_rn(pv, __fadd2_rn(g, u ? make_float2(d4.z, d4.w) : make_float2(d4.x, d4.y)));
          s[e] = pd.x;
          s[e + 1] = pd.y;
          dp[e] = ds.x;
          dp[e + 1] = ds.y;
        }
      }
      if (j > 0) {
        B200FA_WAIT(acc_full, (j - 1) & 1, 0xe20);
        tc_fence_after();
        add_part<kD / 64>(dv, tm + Cfg::kTmemDV + half * (kD / 2), 1.f);
        add_part<kD / 64>(dk, tm + Cfg::kTmemDK + half * (kD / 2), 1.f);
      }
      values_to_tmem(tm + Cfg::kTmemP, s, half);
      values_to_tmem(tm + Cfg::kTmemDS, dp, half);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive_warp(ds_full);
      if ((m0 += kBN) >= p.S) {
        m0 = m_begin;
        ++h;
      }
    }
    if (n > 0) {
      B200FA_WAIT(acc_full, (n - 1) & 1, 0xe21);
      tc_fence_after();
      add_part<kD / 64>(dv, tm + Cfg::kTmemDV + half * (kD / 2), 1.f);
      add_part<kD / 64>(dk, tm + Cfg::kTmemDK + half * (kD / 2), 1.f);
    }
    // (rows past the end are zeros and not masked: with a logsumexp below -88 their probabilities overflow)
    if (n0 + r < p.Sk && (!all_finite(dk) || !all_finite(dv))) *not_finite = 1;
    mbar_arrive_warp(done);
    B200FA_WAIT(done, 0, 0xe30);
    if (*not_finite) {
      if (!fma_rows_dkdv<kD, kDropout>(p, block, smem)) goto teardown;
    } else if (n0 + r < p.Sk) {
      float4* dst_k = reinterpret_cast<float4*>(const_cast<float*>(row_ptr(p.dk, b, hk, n0 + r)) + half * (kD / 2));
      float4* dst_v = reinterpret_cast<float4*>(const_cast<float*>(row_ptr(p.dv, b, hk, n0 + r)) + half * (kD / 2));
#pragma unroll
      for (int i = 0; i < kD / 8; ++i) {
        dst_k[i] = make_float4(dk[4 * i] * p.scale, dk[4 * i + 1] * p.scale, dk[4 * i + 2] * p.scale, dk[4 * i + 3] * p.scale);
        dst_v[i] = make_float4(dv[4 * i], dv[4 * i + 1], dv[4 * i + 2], dv[4 * i + 3]);
      }
    }
  } else if (warp < kConvWarp0 + kConvWarps) {
    // =========================== converters: Q, dO of one tile after the other ===========================
    reg_dealloc<kRegConv>();
    const int tid = threadIdx.x - kConvWarp0 * 32;
    int h = hk * group, m0 = m_begin;   // of the tile being loaded
    auto put = [&](int seq, const float4 (&now)[8]) {
      const int slot = seq % Cfg::kSlots;
      store_box(now, smem + Cfg::kOffStream + slot * Tile::kBytes, Tile::kPlane, tid);
      fence_proxy_async_smem();
      mbar_arrive_warp(&full[slot]);
    };
    auto slot_free = [&](int seq) -> bool {
      return seq < Cfg::kSlots || mbar_wait(&empty[seq % Cfg::kSlots], (seq / Cfg::kSlots - 1) & 1, abort_flag, p.status, 0xe40, p.wait_budget);
    };
    float4 vq[8], vd[8];
    if (n > 0) load_box(vq, p.q, b, h, m0, p.S, 0, tid);
    let_the_dq_kernel_start();
    for (int j = 0; j < n; ++j) {
      load_box(vd, p.dout, b, h, m0, p.S, 0, tid);
      float nl2 = -INFINITY, ndps = 0.f;   // rows past the end, and rows that saw no key: P = 0
      if (tid < kBN && m0 + tid < p.S) {
        const int64_t bh = static_cast<int64_t>(b) * p.Hq + h;
        const float lse = p.lse[bh * p.S + m0 + tid];
        if (lse != -INFINITY) nl2 = -(lse * kLog2e);
        ndps = -__ldcg(p.dpsum + bh * p.Spad + m0 + tid);
      }
      if (!slot_free(2 * j)) goto teardown;
      // The tile's statistics: a slot of theirs is written again four tiles on, when the slot rule above
      // has made sure that the products of the tile three before have completed.
      if (tid < kBN) {
        float* st = sStat + (j % Cfg::kStats) * 2 * kBN + tid;
        st[0] = nl2;
        st[kBN] = ndps;
      }
      put(2 * j, vq);
      if ((m0 += kBN) >= p.S) {
        m0 = m_begin;
        ++h;
      }
      if (j + 1 < n) load_box(vq, p.q, b, h, m0, p.S, 0, tid);
      if (!slot_free(2 * j + 1)) goto teardown;
      put(2 * j + 1, vd);
    }
  } else {
    reg_dealloc<kRegRest>();
    if (warp == kMmaWarp) {
      // =========================== MMA issuer ===========================
      const uint32_t tS = tmem_base + Cfg::kTmemS, tDP = tmem_base + Cfg::kTmemDP, tP = tmem_base + Cfg::kTmemP,
                     tDS = tmem_base + Cfg::kTmemDS, tDV = tmem_base + Cfg::kTmemDV, tDK = tmem_base + Cfg::kTmemDK;
      const uint32_t stream = smem_u32(smem) + Cfg::kOffStream;
      const UmmaDesc dK = umma_desc_split(smem_u32(smem) + Cfg::kOffK, 16, 1024), dV = umma_desc_split(smem_u32(smem) + Cfg::kOffV, 16, 1024);
      const UmmaDesc dCols = umma_desc_split(stream, 16, 1024), dDim = umma_desc_split(stream, kBoxBytes, 1024);
      constexpr uint32_t kSlotLo = umma_off(Tile::kBytes);
      if (n > 0) { B200FA_WAIT_WARP(kv_full, 0, 0xe50); }
      for (int j = -2; j < n; ++j) {
        if (j >= 0) {
          const int q_slot = (2 * j) % Cfg::kSlots, do_slot = (2 * j + 1) % Cfg::kSlots;   // both have been waited for
          B200FA_WAIT_WARP(ds_full, j & 1, 0xe52);
          tc_fence_after();
          issue_dim<kD>(tDV, tP, dDim.lo + do_slot * kSlotLo, dDim.hi);
          umma_commit_elect(&empty[do_slot]);
          issue_dim<kD>(tDK, tDS, dDim.lo + q_slot * kSlotLo, dDim.hi);
          umma_commit_elect(acc_full);
          umma_commit_elect(&empty[q_slot]);
        }
        const int js = j + 2;
        if (js < n) {
          const int seq = 2 * js, q_slot = seq % Cfg::kSlots, do_slot = (seq + 1) % Cfg::kSlots;
          B200FA_WAIT_WARP(&full[q_slot], (seq / Cfg::kSlots) & 1, 0xe53);
          if (js > 0) { B200FA_WAIT_WARP(s_free, (js - 1) & 1, 0xe54); }
          tc_fence_after();
          issue_cols_ss<kD>(tS, dK, dCols.lo + q_slot * kSlotLo, dCols.hi);
          B200FA_WAIT_WARP(&full[do_slot], ((seq + 1) / Cfg::kSlots) & 1, 0xe55);
          tc_fence_after();
          issue_cols_ss<kD>(tDP, dV, dCols.lo + do_slot * kSlotLo, dCols.hi);
          umma_commit_elect(s_full);
        }
      }
    }
  }

teardown:
  tc_fence_before();
  __syncthreads();
  settle_if_aborted(abort_flag);
  if (warp == kMmaWarp) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}
// The dK/dV kernel is launched to start when every block of the dpsum kernel has, and needs that one's results with the
// first tile's statistics.  The dQ kernel does not need the dK/dV kernel's results: it is launched to start as soon as
// every block of that one has seen the dpsum kernel end, and fills the SMs that its last blocks leave idle.  It still ends
// after it: block 0 waits for that, so that what is ordered behind the dQ kernel is ordered behind both.
template <int kD, bool kDropout>
__global__ void __launch_bounds__(kThreads, 1) bwd_dkdv_fp32_kernel(const __grid_constant__ BwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if (status_is_set(p.status)) {
    cudaGridDependencySynchronize();   // (no kernel of a backward ends before the ones launched ahead of it)
    return;
  }
  if ((smem_u32(smem) & 1023u) != 0u) {
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, kStatusOk, 0x414c0003u);
    cudaGridDependencySynchronize();
    return;
  }
  dkdv_block<kD, kDropout>(p, static_cast<int>(blockIdx.x), smem);
}
template <int kD, bool kDropout>
__global__ void __launch_bounds__(kThreads, 1) bwd_dq_fp32_kernel(const __grid_constant__ BwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if (!status_is_set(p.status)) {
    if ((smem_u32(smem) & 1023u) != 0u) {
      if (threadIdx.x == 0 && p.status) atomicCAS(p.status, kStatusOk, 0x414c0004u);
    } else {
      dq_block<kD, kDropout>(p, static_cast<int>(blockIdx.x), smem);
    }
  }
  if (blockIdx.x == 0) cudaGridDependencySynchronize();
}
#undef B200FA_WAIT
#undef B200FA_WAIT_WARP

// dpsum = rowsum(dO * O).  A row is D / 4 lanes of 16 bytes; a thread issues the loads of four rows before it
// adds any of them up, and a block lies inside one (b, h).
template <int kD>
struct PreF32Cfg {
  static constexpr int kLanes = kD / 4, kRowsPerWarp = 32 / kLanes, kRows = 4, kBlockRows = 8 * kRowsPerWarp * kRows;
};
template <int kD>
__global__ void __launch_bounds__(256) dpsum_fp32_kernel(const BwdParams p) {
  using Cfg = PreF32Cfg<kD>;
  cudaTriggerProgrammaticLaunchCompletion();
  const int lane = threadIdx.x & 31, li = lane % Cfg::kLanes;
  const int per_head = (p.S + Cfg::kBlockRows - 1) / Cfg::kBlockRows;
  const int bh = static_cast<int>(blockIdx.x) / per_head, b = bh / p.Hq, h = bh - b * p.Hq;
  const int s0 = (static_cast<int>(blockIdx.x) - bh * per_head) * Cfg::kBlockRows +
                 (threadIdx.x >> 5) * Cfg::kRowsPerWarp * Cfg::kRows + lane / Cfg::kLanes;
  float4 o[Cfg::kRows], g[Cfg::kRows];
#pragma unroll
  for (int u = 0; u < Cfg::kRows; ++u) {
    const int s = s0 + u * Cfg::kRowsPerWarp;
    o[u] = g[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (s < p.S) {
      o[u] = reinterpret_cast<const float4*>(row_ptr(p.out, b, h, s))[li];
      g[u] = reinterpret_cast<const float4*>(row_ptr(p.dout, b, h, s))[li];
    }
  }
#pragma unroll
  for (int u = 0; u < Cfg::kRows; ++u) {
    float acc = fmaf(o[u].x, g[u].x, o[u].y * g[u].y) + fmaf(o[u].z, g[u].z, o[u].w * g[u].w);
#pragma unroll
    for (int off = Cfg::kLanes / 2; off >= 1; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    const int s = s0 + u * Cfg::kRowsPerWarp;
    if (li == 0 && s < p.S) p.dpsum[static_cast<int64_t>(bh) * p.Spad + s] = acc;
  }
}

// cudaFuncSetAttribute once per device and kernel (`once` and `result` are statics of the function template
// that names the kernel), safe against concurrent first calls
template <typename Kernel>
cudaError_t allow_dynamic_smem(Kernel kern, int bytes, std::once_flag (&once)[64], cudaError_t (&result)[64]) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  std::call_once(once[dev], [&] { result[dev] = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); });
  return result[dev];
}

template <int kD, bool kDropout>
cudaError_t launch_fwd(const FwdParams& p, cudaStream_t stream) {
  auto kern = fwd_fp32_kernel<kD, kDropout>;
  static std::once_flag once[64];
  static cudaError_t result[64];
  constexpr int smem = FwdF32Cfg<kD>::kSmemBytes;
  const cudaError_t e = allow_dynamic_smem(kern, smem, once, result);
  if (e != cudaSuccess) return e;
  const int64_t blocks = static_cast<int64_t>(p.B) * p.Hq * ((p.Sq + kBM - 1) / kBM);
  kern<<<static_cast<unsigned>(blocks), kThreads, smem, stream>>>(p);
  return cudaGetLastError();
}

template <int kD, bool kDropout>
cudaError_t launch_bwd(const BwdParams& p, cudaStream_t stream) {
  auto k1 = bwd_dkdv_fp32_kernel<kD, kDropout>;
  auto k2 = bwd_dq_fp32_kernel<kD, kDropout>;
  static std::once_flag once1[64], once2[64];
  static cudaError_t result1[64], result2[64];
  cudaError_t e;
  if ((e = allow_dynamic_smem(k1, DkdvF32Cfg<kD>::kSmemBytes, once1, result1)) != cudaSuccess) return e;
  if ((e = allow_dynamic_smem(k2, DqF32Cfg<kD>::kSmemBytes, once2, result2)) != cudaSuccess) return e;
  const int64_t pre_blocks = static_cast<int64_t>(p.B) * p.Hq * ((p.S + PreF32Cfg<kD>::kBlockRows - 1) / PreF32Cfg<kD>::kBlockRows);
  dpsum_fp32_kernel<kD><<<static_cast<unsigned>(pre_blocks), 256, 0, stream>>>(p);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  const int64_t kv_blocks = static_cast<int64_t>(p.B) * p.Hkv * ((p.Sk + kBM - 1) / kBM);
  const int64_t q_blocks = static_cast<int64_t>(p.B) * p.Hq * ((p.S + kBM - 1) / kBM);
  e = launch_early(k1, dim3(static_cast<unsigned>(kv_blocks)), kThreads, DkdvF32Cfg<kD>::kSmemBytes, stream, true, p);
  if (e != cudaSuccess) return e;
  return launch_early(k2, dim3(static_cast<unsigned>(q_blocks)), kThreads, DqF32Cfg<kD>::kSmemBytes, stream, true, p);
}

// Few keys at D = 128: the fp32 FMA kernels have less to set up and smaller tiles, and lose as soon as they run in waves.
// B200, us, FMA kernels against these: B1 Hq32 Sq86 12.0 / 13.6, 98 keys B16 Hq24 73.6 / 41.7.
// At D = 64 they would save 1-3 us of 6-14 below 96 keys while they fit at once (B2 Hq12 Sq1061 Sk92 9.5 against 16.3; in
// waves they lose, B16 H8 Sq1000 Sk77 121 / 66), but the backward there is on the tensor cores at any length, and a forward
// and a backward whose scores have different errors give gradients up to eight times further from float64 than two of one
// kind, where keys share a large component.
bool few_keys(const FwdParams& p) {
  const int64_t keys = p.causal ? std::min<int64_t>(p.Sk, static_cast<int64_t>(p.Sq) + p.causal_off) : p.Sk;   // that anyone sees
  return p.D == 128 && keys <= 128 && p.whole_heads * ((p.Sq + 31) / 32) <= 148;
}

}  // namespace

// Relative errors (2-norm, the worst of out / dQ / dK / dV, these kernels against the fp32 FMA ones): B4 H12 S1024 D64
// causal 3.5e-7 / 7.8e-7, B1 Hq4 Hkv2 S4096 D64 causal 3.8e-7 / 1.9e-6, Sq64 Sk16384 D64 5.8e-7 / 2.3e-6; out alone at
// D = 128: S777 2.6e-7 / 5.6e-7, Sq130 Sk8192 2.7e-7 / 1.7e-6.  Over normal values of spread 0.5 to 1 and 128 to 4096 keys,
// in terms of the FMA kernels' error: out 0.18-0.55, dQ 0.41-0.86, dK 0.30-0.81, dV 0.27-0.71, lse 0.96-1.07 (1.00 on average).
// Times (us, B200): B4 H12 S1024 D64 causal forward 163 -> 56, backward 563 -> 155; B2 Hq16 Hkv4 S1024 D128 unmasked forward
// 488 -> 130; B2 H4 S256 D64 causal 12.8 -> 12.8 and 41 -> 22.4.
cudaError_t launch_fwd_fp32(const FwdParams& p, cudaStream_t stream, int* launches) {
  if (few_keys(p)) return launch_fwd_simt(p, kF32, stream, launches);
  const bool drop = p.drop.threshold != 0;
  const cudaError_t e = p.D == 64 ? (drop ? launch_fwd<64, true>(p, stream) : launch_fwd<64, false>(p, stream))
                                  : (drop ? launch_fwd<128, true>(p, stream) : launch_fwd<128, false>(p, stream));
  if (e == cudaSuccess && launches) *launches += 1;
  return e;
}

// At any length.  B200, us, FMA kernels against these: one to 64 heads 14-16 / 10-13 at 16 to 64 rows and keys, 73 / 34 at Sq96
// Sk1024; 256 heads 97 / 55 at 128 rows and keys; 1024 heads 137 / 135 at 64.  The FMA kernels are faster only for up to 32 rows
// and keys of 75 to 443 heads (296 heads: 22 / 33), where a second wave of 128-row blocks costs more than the blocks do;
// a rule on heads would give a piece of a batch other bits than the whole, and the call's host side takes 200 us.
cudaError_t launch_bwd_fp32(const BwdParams& p, cudaStream_t stream, int* launches) {
  const cudaError_t e = p.drop.threshold != 0 ? launch_bwd<64, true>(p, stream) : launch_bwd<64, false>(p, stream);
  if (e == cudaSuccess && launches) *launches += 3;
  return e;
}

}  // namespace b200fa
