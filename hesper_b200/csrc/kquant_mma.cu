// kquant_mma.cu -- batched (16 tokens or more) Q4_K / Q8_0 product with the dequantiser fused into
// the tensor-core kernel: the weights go from their blocks to f16 in registers and from there
// straight into TENSOR MEMORY as the A operand of tcgen05.mma kind::f16; the f16 image of the
// tensor never exists in global memory.
//
// Same contract as the streaming kernels (Q4_K: w = d*sc*q - dmin*m, Q8_0: w = d*q; f32
// activations in, f32 out; the reference's batched counterparts are the M>1 paths of
// Hesper/Layers/Linear.lean:1152-1760,5973-6177).  Weights AND activations are rounded to f16
// (2^-11 each): measured error ~4e-4 of max|y|, bar 1e-3.
//
// What bounds it: at 64 tokens instruction issue of the SMs at work (81 % of the slots; 4.9 instructions
// per weight, two of them the dequantiser's arithmetic, the rest loads, scales, tensor-memory stores,
// barriers and polling), at 256 tokens the tensor pipe (M=128, N=256, K=16 in 138 cycles).  Either
// way only when every SM works, so the work is dealt in units of (row tile of 128, super-block of 256 weights):
//   * whole waves of row tiles go one tile to a CTA (W per CTA, results stored directly);
//   * the R row tiles left over are cut along K into runs of `upc` consecutive units, one run
//     per CTA.  A run that does not cover its tile leaves an f32 partial in the context's
//     scratch and a small second kernel adds a tile's partials in K order (deterministic; adding
//     them in this kernel by the last part to arrive was slower: the fence in front of the
//     ticket waits for the CTA's stores, 43 against 28 us at K=10240 N=2560, 256 tokens).
//     160 tiles of a 10240-row gate/up pair so take 11 super-block times on 148 SMs instead of
//     20, the 20 tiles of a 2560-row down projection 6 instead of 40.
// Warps with fixed roles:
//   16 or 24   dequantise, in groups of 8 that take the A stages in turn; a thread owns one row and
//              64 weights of every 128 and stores them with tcgen05.st.  The first 16 also run
//              the epilogue of a finished tile, after they have refilled the A stages for the
//              next one;
//   one        weights: 2-D tensor-map TMA boxes of 64 rows x 256 weights, a ring of 2 to 6 tiles;
//   one        activations: bulk copies of a super-block's tiles (f16, operand layout written by
//              the staging kernel);
//   one        an elected thread issues the MMAs (M=128, N=NT tokens, K=16).
// A gate/up pair is one launch: a tile holds 64 gate rows and the 64 up rows of the same outputs,
// dealt to the tensor-memory lanes so that a gate lane's up value sits 16 lanes further in the
// same warp (one shuffle per two tokens in the epilogue).
// Every wait is bounded; on expiry the kernel still releases its tensor memory.
#include <cuda_fp16.h>

#include "tcgen05.cuh"

namespace hb {

constexpr int kQmRows = 128;          // weight rows per tile = MMA M
constexpr int kQmMaxSeg = 4;          // tensors one launch multiplies by the same activations

// NT tokens per pass = MMA N; a unit is the bytes of 256 weights (one Q4_K super-block, eight
// Q8_0 blocks).
template <int NT, int FMT>
struct QmCfg {
  static constexpr int kUnit = FMT == 12 ? 144 : 272;
  static constexpr int kPkBytes = kQmRows * kUnit;          // 18 / 34 KB
  // kind::f16: D = f32, A and B f16, both K-major, N = NT, M = 128
  static constexpr uint32_t kIdesc =
      (1u << 4) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(kQmRows >> 4) << 24);
  static constexpr bool kSums = FMT == 12;                  // sub-block sums as extra K columns
  // A stages in tensor memory (two weights per column) hold a whole super-block, or half of one
  // where a 256-token accumulator leaves no room: a stage costs its warps two barriers, a fence
  // and the wait for their stores, ~400 cycles whatever it holds
  static constexpr int kAParts = NT == 256 ? 2 : 1;         // stages per super-block
  static constexpr int kACols = 128 / kAParts;
  static constexpr int kAStages = NT == 128 ? 2 : 3;
  static constexpr int kA0 = NT;                            // after the accumulator
  static constexpr int kE0 = kA0 + kAStages * kACols;       // columns of the min residues:
  static constexpr int kESlots = kSums ? 8 : 0;             //   8 per super-block
  // staged bytes of a super-block: four blocks of [NT rows][64 f16], then [NT rows][16 f16]
  static constexpr int kSumBytes = kSums ? NT * 32 : 0;
  static constexpr int kSbBytes = NT * 512 + kSumBytes;
  // activation stages: a super-block, or a quarter of one at 256 tokens; the last brings the sums
  static constexpr int kBParts = NT == 256 ? 4 : 1;
  static constexpr int kBPart = NT * 512 / kBParts;         // 32 / 64 / 32 KB
  static constexpr int kBBytes = kBPart + kSumBytes;
  static constexpr int kBStages = NT == 64 ? 3 : (NT == 128 ? 2 : 4);
  static constexpr int kPkStages = FMT == 12 ? (NT == 64 ? 6 : (NT == 128 ? 4 : 3)) : (NT == 64 ? 3 : 2);
  // dequantising warps, in groups of 8 that take the stages in turn: filling one is a chain of
  // 1000 to 2000 cycles of which a warp issues a fifth
  static constexpr int kGroups = NT == 64 ? 3 : 2;
  static constexpr int kExpWarps = 8 * kGroups;
  static constexpr int kThreads = (kExpWarps + 3) * 32;
  static constexpr int kSmem = 2048 + kPkStages * kPkBytes + kBStages * kBBytes;
  static_assert(kE0 + kESlots * 8 <= 512, "tensor memory columns");
  static_assert(kSmem <= 232448, "shared memory budget of one CTA");
};

struct QmSeg {
  const float* residual;  // nullable
  float* y;               // y[m * ldy + row]
  long ldy;
  int N;
  int tile0;              // first row tile of this tensor in the launch
};

// How the tiles are dealt to the CTAs (see the head of the file).
struct QmDeal {
  int W;      // whole tiles per CTA: tile w * grid + cta
  int R;      // tiles left over, numbered from W * grid
  int nb;     // units (super-blocks) per tile
  int upc;    // units of the left-over tiles per CTA: [cta * upc, (cta + 1) * upc)
};

struct QmParams {
  CUtensorMap tmap[kQmMaxSeg];  // blocks as [N rows][rowbytes], boxes of 64 rows x one unit
  QmSeg seg[kQmMaxSeg];
  int nseg;
  int glu;                // seg 0 = gate, seg 1 = up; y = gelu_tanh(gate) * up into seg 0's y
  QmDeal deal;
  const uint8_t* xb;      // staged activations: kSbBytes per super-block
  const float* rowscale;  // [NT] power of two each token's row was divided by before rounding
  int M;
  float* part;            // [cta][2][NT / 4][128 lanes][4 tokens] partial sums of left-over tiles
  uint32_t* status;
};

// 0.5*g*(1+tanh(t)), t = sqrt(2/pi)*(g+0.044715 g^3), the gate factor of the GeGLU
// (Hesper/Layers/FusedFFNSpec.lean:42-45), as g * sigmoid(2t): the same function without the
// cancellation of 1 + tanh at negative t, and a third of tanhf's instructions (the epilogue of a
// 256-token tile evaluates 16384 of them).  t -> -inf: exp overflows to inf, the result is -0.
__device__ __forceinline__ float glu_gate(float g) {
  const float t2 = 1.5957691216057308f * (g + 0.044715f * g * g * g);
  return __fdividef(g, 1.0f + __expf(-t2));
}

__device__ __forceinline__ __half2 as_h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }
__device__ __forceinline__ uint32_t as_u32(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }

// 32 nibble bytes of a chunk (two sub-blocks of 32 weights: low and high nibbles) -> 64 f16.
// Everything stays in packed f16 and only one step rounds: LOP3 completes two nibbles to the
// f16 1024 + q (low) or 1024 + 16 q (high), one HFMA2 turns them into the integers sc * q (at
// most 945: exact), one HFMA2 forms d * (sc q) - c with c = dmin * m rounded to f16.  What c lost,
// e = dmin * m - c, is not dropped: it goes into the product as sixteen further K columns per
// super-block (e of its 8 sub-blocks against the sub-blocks' activation sums), so the weights
// carry the one rounding of the f32 formula and nothing else.  Two instructions per two weights
// and step instead of five through f32 (I2F / FFMA / pack).
// The pairs come out as bytes {0, 2}, {1, 3} of every word; the activations are staged in the
// same order.  HI: the high nibbles.
template <bool HI>
__device__ __forceinline__ void q4k_expand(const uint32_t (&q)[8], __half2 d, __half2 mul, __half2 add,
                                           __half2 c, uint32_t (&o)[16]) {
  constexpr uint32_t kMask = HI ? 0x00F000F0u : 0x000F000Fu;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t t0 = (q[i] & kMask) | 0x64006400u, t1 = ((q[i] >> 8) & kMask) | 0x64006400u;
    o[2 * i] = as_u32(__hfma2(d, __hfma2(as_h2(t0), mul, add), c));
    o[2 * i + 1] = as_u32(__hfma2(d, __hfma2(as_h2(t1), mul, add), c));
  }
}

// The same by the f32 formula: dmin * m may lie outside f16 although the weight does not.
template <bool HI>
__device__ __forceinline__ void q4k_expand_f32(const uint32_t (&q)[8], float d, float c, uint32_t (&o)[16]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t t = HI ? q[i] >> 4 : q[i];
    auto w = [&](int sh) { return fmaf(d, (float)(t >> sh & 15u), c); };
    o[2 * i] = as_u32(__floats2half2_rn(w(0), w(16)));
    o[2 * i + 1] = as_u32(__floats2half2_rn(w(8), w(24)));
  }
}

// Four int8 times d, rounded once to f16: bytes biased to 1024 + (q + 128), the bias taken off
// exactly, then an f16 product (d is an f16, q an integer: the exact product is rounded once).
// Pairs {0, 2}, {1, 3} as in q4k_expand.
__device__ __forceinline__ void q80_word(uint32_t w, __half2 d, uint32_t& lo, uint32_t& hi) {
  const uint32_t x = w ^ 0x80808080u;
  const uint32_t a = __byte_perm(x, 0x64646464u, 0x4240), b = __byte_perm(x, 0x64646464u, 0x4341);
  const __half2 bias = __floats2half2_rn(1152.f, 1152.f);
  lo = as_u32(__hmul2(__hsub2(as_h2(a), bias), d));
  hi = as_u32(__hmul2(__hsub2(as_h2(b), bias), d));
}

// One stretch of work of a CTA: units [b0, b0 + n) of a tile.
struct QmJob {
  int tile, b0, n, slot;  // slot: -1 = the whole tile, else which of the CTA's two partials
};
__device__ __forceinline__ int qm_jobs(const QmDeal& d) {
  const int u0 = (int)blockIdx.x * d.upc, u1 = min(u0 + d.upc, d.R * d.nb);
  if (u0 >= u1) return d.W;
  return d.W + ((u1 - 1) / d.nb - u0 / d.nb + 1);
}
__device__ __forceinline__ QmJob qm_job(const QmDeal& d, int j) {
  if (j < d.W) return {(int)blockIdx.x + j * (int)gridDim.x, 0, d.nb, -1};
  const int k = j - d.W;
  const int u0 = (int)blockIdx.x * d.upc, u1 = min(u0 + d.upc, d.R * d.nb);
  const int t = u0 / d.nb + k;
  const int lo = max(u0, t * d.nb), hi = min(u1, (t + 1) * d.nb);
  return {d.W * (int)gridDim.x + t, lo - t * d.nb, hi - lo, hi - lo == d.nb ? -1 : k};
}

// ---- staging of the activations -----------------------------------------------------------
//
// One CTA per token row: optional x' = base + rmsnorm(x) * pre_gamma (x' also written out), optional
// RMSNorm * gamma, the row divided by a power of two that brings its largest magnitude into
// [2^13, 2^14) (f16 has 5 exponent bits: an activation above 65504 would round to infinity, one
// below 6e-5 lose bits; the product's epilogue multiplies the scale back), rounded to f16 and laid
// out as the MMA's B operand: per super-block four blocks [row / 8][k / 8][row % 8][8 k] of 64
// elements and, for Q4_K, [row / 8][2][row % 8][8] with the sums of the 8 sub-blocks / 32 (the
// second half zero).  The four bytes of a weight word pair up as {0, 2}, {1, 3}: so do the k here.
// Latency is all there is to it (a row, three block-wide reductions at most), so the row stays
// in registers from its one read and the norm weights are fetched before the wait.
//
// I8: the operand of the few-token kernel instead (kquant_sb.cu).  Every 32 elements become 16-bit
// integers of their own scale, x ~ dx * (256*hi + lo) with hi and lo signed bytes, laid out as
// mma.sync's B fragments per (sub-block, 8 tokens): lane 4 * (token % 8) + t holds {hi, hi, lo, lo}
// of elements 8t..8t+7; behind them {dx, dx, sum, sum} of two tokens per entry.  Rows past the last
// token are zero.
struct QmStage {
  const float *x, *gamma, *pre_base, *pre_gamma;
  float* pre_out;
  float eps;
  int K;
  uint8_t* xb;
  size_t sb_bytes;   // bytes of a super-block
  int sums_off;      // where its sums start, 0: none
  float* rowscale;
  int M, ntl;        // I8 only: tokens, token columns / 8
};

template <int G, bool I8>
__global__ void __launch_bounds__(1024) kq_stage_kernel(const __grid_constant__ QmStage p) {
  __shared__ double red[2][32];
  __shared__ float redf[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int m = blockIdx.x, n8 = p.K >> 3;
  float g[G][8], pg[G][8], v[G][8];
  auto load8 = [&](float (&d)[8], const float* src, int i, bool ro) {
    if (ro && (reinterpret_cast<uintptr_t>(src) & 15)) {  // norm weights may sit anywhere
#pragma unroll
      for (int e = 0; e < 8; ++e) d[e] = __ldg(src + 8 * i + e);
      return;
    }
    const float4* s4 = reinterpret_cast<const float4*>(src) + 2 * i;
    const float4 a = ro ? __ldg(s4) : __ldcg(s4), b = ro ? __ldg(s4 + 1) : __ldcg(s4 + 1);
    d[0] = a.x; d[1] = a.y; d[2] = a.z; d[3] = a.w;
    d[4] = b.x; d[5] = b.y; d[6] = b.z; d[7] = b.w;
  };
  pdl_trigger();
#pragma unroll
  for (int j = 0; j < G; ++j) {
    const int i = tid + j * blockDim.x;
    if (i < n8 && p.gamma) load8(g[j], p.gamma, i, true);
    if (i < n8 && p.pre_gamma) load8(pg[j], p.pre_gamma, i, true);
  }
  pdl_wait();
  const bool real = !I8 || m < p.M;  // I8: the whole CTA of a row past the last token stays at zero
#pragma unroll
  for (int j = 0; j < G; ++j) {
    const int i = tid + j * blockDim.x;
#pragma unroll
    for (int e = 0; e < 8; ++e) v[j][e] = 0.f;
    if (real && i < n8) load8(v[j], p.x + (size_t)m * p.K, i, false);
  }
  auto row_rinv = [&](double* scr) {  // 1 / rms of the row held in v (block-wide)
    double ss = 0.0;
#pragma unroll
    for (int j = 0; j < G; ++j)
#pragma unroll
      for (int e = 0; e < 8; ++e) ss += (double)v[j][e] * v[j][e];
    ss = warp_sum(ss);
    if (lane == 0) scr[warp] = ss;
    __syncthreads();
    ss = warp_sum(lane < nwarps ? scr[lane] : 0.0);
    return (float)(1.0 / sqrt(ss / (double)p.K + (double)p.eps));
  };
  if (real && p.pre_gamma) {
    float b[G][8];
#pragma unroll
    for (int j = 0; j < G; ++j) {
      const int i = tid + j * blockDim.x;
      if (i < n8) load8(b[j], p.pre_base + (size_t)m * p.K, i, false);
    }
    const float r1 = row_rinv(red[0]);
#pragma unroll
    for (int j = 0; j < G; ++j) {
      const int i = tid + j * blockDim.x;
      if (i < n8) {
#pragma unroll
        for (int e = 0; e < 8; ++e)
          v[j][e] = __fadd_rn(b[j][e], __fmul_rn(__fmul_rn(v[j][e], r1), pg[j][e]));
        float4* og = reinterpret_cast<float4*>(p.pre_out + (size_t)m * p.K) + 2 * i;
        og[0] = make_float4(v[j][0], v[j][1], v[j][2], v[j][3]);
        og[1] = make_float4(v[j][4], v[j][5], v[j][6], v[j][7]);
      }
    }
  }
  if (real && p.gamma) {
    const float rinv = row_rinv(red[1]);
#pragma unroll
    for (int j = 0; j < G; ++j)
      if (tid + j * (int)blockDim.x < n8) {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[j][e] = __fmul_rn(__fmul_rn(v[j][e], rinv), g[j][e]);
      }
  }
  if constexpr (I8) {
#pragma unroll
    for (int j = 0; j < G; ++j) {
      const int i = tid + j * blockDim.x;
      float amax = 0.f, sum = 0.f;  // of the four lanes that share 32 elements
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        amax = fmaxf(amax, fabsf(v[j][e]));
        sum += v[j][e];
      }
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
      }
      if (i >= n8) continue;
      const float inv = amax > 0.f ? 32512.0f / amax : 0.f;
      uint32_t q[8];  // q + 128 = 256 * hi + (lo + 128): hi is its byte 1, lo its byte 0 ^ 0x80
#pragma unroll
      for (int e = 0; e < 8; ++e) q[e] = (uint32_t)(__float2int_rn(v[j][e] * inv) + 128);
      auto bytes = [&](int a, uint32_t sel) {
        return __byte_perm(__byte_perm(q[a], q[a + 1], sel), __byte_perm(q[a + 2], q[a + 3], sel), 0x5410);
      };
      const int sj = (i >> 2) & 7, t = i & 3, nt = m >> 3, g = m & 7;
      uint8_t* sb = p.xb + (size_t)(i >> 5) * p.sb_bytes;
      *reinterpret_cast<uint4*>(sb + ((sj * p.ntl + nt) * 32 + 4 * g + t) * 16) =
          make_uint4(bytes(0, 0x0051), bytes(4, 0x0051), bytes(0, 0x0040) ^ 0x80808080u,
                     bytes(4, 0x0040) ^ 0x80808080u);
      float* tab = reinterpret_cast<float*>(sb + p.ntl * 4096 + ((sj * p.ntl + nt) * 4 + (g >> 1)) * 16) + (g & 1);
      // Q4_K multiplies the high nibbles in place: their 16 is taken off here
      if (t == 0) tab[0] = amax / 32512.0f * (p.sums_off && (sj & 1) ? 0.0625f : 1.f);
      if (t == 1) tab[2] = sum;
    }
    return;
  }
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < G; ++j)
#pragma unroll
    for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(v[j][e]));  // groups past K hold zeros
  amax = warp_max(amax);
  if (lane == 0) redf[warp] = amax;
  __syncthreads();
  amax = warp_max(lane < nwarps ? redf[lane] : 0.f);
  int ex = 13;  // an all-zero (or non-finite) row keeps scale 1
  if (amax > 0.f && amax <= 3.0e38f) ex = min(max(ilogbf(amax), -100), 120);
  if (tid == 0) p.rowscale[m] = ldexpf(1.f, ex - 13);
  const float inv_s = ldexpf(1.f, 13 - ex);
#pragma unroll
  for (int j = 0; j < G; ++j) {
    const int i = tid + j * blockDim.x;
    float sum = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      v[j][e] *= inv_s;  // exact: a power of two
      sum += v[j][e];
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if (i >= n8) continue;
    uint8_t* sb = p.xb + (size_t)(i >> 5) * p.sb_bytes;
    uint4 o;
    o.x = as_u32(__floats2half2_rn(v[j][0], v[j][2]));
    o.y = as_u32(__floats2half2_rn(v[j][1], v[j][3]));
    o.z = as_u32(__floats2half2_rn(v[j][4], v[j][6]));
    o.w = as_u32(__floats2half2_rn(v[j][5], v[j][7]));
    // four blocks of NT rows x 128 bytes: sums_off (or sb_bytes) is their total
    const size_t blk = (p.sums_off ? (size_t)p.sums_off : p.sb_bytes) >> 2;
    *reinterpret_cast<uint4*>(sb + ((i & 31) >> 3) * blk + (m >> 3) * 1024 + (i & 7) * 128 + (m & 7) * 16) = o;
    if (p.sums_off) {
      uint8_t* sd = sb + p.sums_off + (m >> 3) * 256 + (m & 7) * 16;
      if ((i & 3) == 0)
        *reinterpret_cast<__half*>(sd + ((i & 31) >> 2) * 2) = __float2half_rn(sum * 0.03125f);
      if ((i & 31) == 1) *reinterpret_cast<uint4*>(sd + 128) = make_uint4(0, 0, 0, 0);
    }
  }
}

template <int NT, int FMT>
__global__ void __launch_bounds__(QmCfg<NT, FMT>::kThreads, 1) kq_mma_kernel(const __grid_constant__ QmParams p) {
  using Cfg = QmCfg<NT, FMT>;
  constexpr int kPkStages = Cfg::kPkStages, kPkBytes = Cfg::kPkBytes, kUnit = Cfg::kUnit;
  constexpr int kAStages = Cfg::kAStages, kAParts = Cfg::kAParts, kACols = Cfg::kACols, kA0 = Cfg::kA0;
  constexpr int kBStages = Cfg::kBStages, kBParts = Cfg::kBParts, kBBytes = Cfg::kBBytes;
  constexpr int kGroups = Cfg::kGroups;
  // a box dimension holds at most 256 elements: the 272-byte Q8_0 unit is mapped as 68 words
  constexpr int kBoxX = FMT == 12 ? 144 : 68;
  constexpr int kEpiWarps = 16;
  constexpr int kPkWarp = Cfg::kExpWarps, kActWarp = kPkWarp + 1, kMmaWarp = kPkWarp + 2;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);

  uint64_t* pk_full = reinterpret_cast<uint64_t*>(smem);  // [kPkStages] two boxes landed
  uint64_t* pk_free = pk_full + kPkStages;                // [kPkStages] every expander warp left it
  uint64_t* a_full = pk_free + kPkStages;    // [kAStages] stored by a group's 8 warps
  uint64_t* a_free = a_full + kAStages;      // [kAStages] the MMAs that read it have retired
  uint64_t* b_full = a_free + kAStages;      // [kBStages] activations landed
  uint64_t* b_free = b_full + kBStages;      // [kBStages]
  uint64_t* acc_full = b_free + kBStages;    // a tile's products are complete
  uint64_t* acc_free = acc_full + 1;         // the epilogue has read them
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + 1);
  float* rs_s = reinterpret_cast<float*>(smem + 1024);  // [NT] row scales
  uint8_t* pk = smem + 2048;
  uint8_t* bstg = pk + kPkStages * kPkBytes;

  if (tid == 0) {
    for (int i = 0; i < kPkStages; ++i) {
      mbar_init(&pk_full[i], 1);
      mbar_init(&pk_free[i], 8 * kAParts);
    }
    for (int i = 0; i < kAStages; ++i) {
      mbar_init(&a_full[i], 8);
      mbar_init(&a_free[i], 1);
    }
    for (int i = 0; i < kBStages; ++i) {
      mbar_init(&b_full[i], 1);
      mbar_init(&b_free[i], 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_free, kEpiWarps);
    fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
        smem_u32(tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_before_sync();
  __syncthreads();
  tc_after_sync();
  // All 512 columns are this CTA's, so the allocation starts at column 0: a constant base keeps
  // the MMA warp's addresses in the uniform datapath.
  constexpr uint32_t tmem = 0;
  const int njobs = qm_jobs(p.deal);
  bool ok = true;
  pdl_trigger();

  if (warp == kPkWarp) {
    // ================= weights: constant, so no wait on the previous kernel =====================
    // ... as long as no slot has to be freed by way of a product (bounded waits, see tc_wait)
    const uint64_t pol = policy_evict_first();
    constexpr int kAhead = kPkStages + kAStages / kAParts;
    int nth = 0;
    TcRing<kPkStages> r;
    for (int j = 0; j < njobs && ok; ++j) {
      const QmJob job = qm_job(p.deal, j);
      int si = 0;
      if (!p.glu) {
#pragma unroll
        for (int i = 1; i < kQmMaxSeg; ++i)
          if (i < p.nseg && job.tile >= p.seg[i].tile0) si = i;
      }
      const CUtensorMap* tm0 = &p.tmap[si];
      const CUtensorMap* tm1 = p.glu ? &p.tmap[1] : tm0;
      const int y0 = p.glu ? job.tile * 64 : (job.tile - p.seg[si].tile0) * kQmRows;
      const int y1 = p.glu ? y0 : y0 + 64;
      int x = job.b0 * kBoxX;
      for (int b = 0; b < job.n; ++b, x += kBoxX, r.advance()) {
        if (nth++ == kAhead) pdl_wait();
        ok = tc_wait_w(&pk_free[r.i], r.phase ^ 1, p.status);
        if (!ok) break;
        if (tc_elect()) {
          mbar_arrive_expect_tx(&pk_full[r.i], kPkBytes);
          uint8_t* dst = pk + (size_t)r.i * kPkBytes;
          tc_tma_box_2d(dst, tm0, x, y0, &pk_full[r.i], pol);
          tc_tma_box_2d(dst + kPkBytes / 2, tm1, x, y1, &pk_full[r.i], pol);
        }
        __syncwarp();
      }
    }
  } else if (warp == kActWarp) {
    // ================= activations: written by the kernel before this one =======================
    pdl_wait();
    TcRing<kBStages> r;
    for (int j = 0; j < njobs && ok; ++j) {
      const QmJob job = qm_job(p.deal, j);
      const uint8_t* src = p.xb + (size_t)job.b0 * Cfg::kSbBytes;
      for (int s = 0; s < job.n && ok; ++s) {
#pragma unroll
        for (int h = 0; h < kBParts; ++h, r.advance()) {
          const uint32_t bytes = h == kBParts - 1 ? kBBytes : Cfg::kBPart;
          ok = tc_wait_w(&b_free[r.i], r.phase ^ 1, p.status);
          if (!ok) break;
          if (tc_elect()) {
            mbar_arrive_expect_tx(&b_full[r.i], bytes);
            bulk_g2s(bstg + (size_t)r.i * kBBytes, src, bytes, &b_full[r.i]);
          }
          __syncwarp();
          src += bytes;
        }
      }
    }
  } else if (warp == kMmaWarp) {
    // ================= MMA issue: the whole warp runs the loop, one lane issues =================
    // Nothing in the loop's control flow depends on a wait's outcome: ring positions stay provably
    // uniform, so the addresses are computed in the uniform datapath instead of being moved there
    // for every MMA (the warp shares its scheduler with six busy ones).  After an expired wait
    // the products run on whatever is there; the status word says so.
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      if (!mbar_try_wait(bar, parity) && ok) ok = tc_wait_slow(smem_u32(bar), parity, p.status);
    };
    pdl_wait();  // the activations come behind it: the waits below are bounded by this kernel's own work
    TcRing<kAStages> ra;
    TcRing<kBStages> rb;
    uint32_t eslot = 0, dphase = 0;
    const uint32_t b0 = tc_desc_lo(smem_u32(bstg), 128);
    for (int j = 0; j < njobs; ++j, dphase ^= 1) {
      const int nu = qm_job(p.deal, j).n;
      wait(acc_free, dphase ^ 1);
      uint32_t accum = 0;
      for (int u = 0; u < nu; ++u) {
#pragma unroll
        for (int ap = 0; ap < kAParts; ++ap, ra.advance()) {
          wait(&a_full[ra.i], ra.phase);
          const uint32_t a_t = tmem + kA0 + ra.i * kACols;
          constexpr int kPer = kBParts / kAParts;
#pragma unroll
          for (int bp = 0; bp < kPer; ++bp, rb.advance()) {
            wait(&b_full[rb.i], rb.phase);
            tc_after_sync();
            const uint32_t bdesc = b0 + rb.i * (kBBytes >> 4);
            constexpr int kMma = 16 / kBParts;  // K = 16 per instruction: 8 columns of A
#pragma unroll
            for (int m = 0; m < kMma; ++m) {
              tc_mma_f16_ta_w<tc_desc_hi(1024), Cfg::kIdesc>(
                  tmem, a_t + (bp * kMma + m) * 8,
                  bdesc + (((m >> 2) * (NT * 128) + (m & 3) * 256) >> 4), accum);
              accum = 1;
            }
            if constexpr (Cfg::kSums)
              if (ap == kAParts - 1 && bp == kPer - 1) {  // residues of the super-block's mins
                tc_mma_f16_ta_w<tc_desc_hi(256), Cfg::kIdesc>(tmem, tmem + Cfg::kE0 + eslot * 8,
                                                              bdesc + (Cfg::kBPart >> 4), 1u);
                eslot = (eslot + 1) % Cfg::kESlots;
              }
            tc_commit_w(&b_free[rb.i]);
          }
          tc_commit_w(&a_free[ra.i]);
        }
      }
      tc_commit_w(acc_full);
    }
  } else {
    // ================= dequantise into tensor memory, epilogue ==================================
    const int q = warp & 3, c2 = (warp >> 2) & 1, grp = warp >> 3;  // lane quarter, which 64 of
                                                                    // every 128 weights, group
    // row of the tile that this tensor-memory lane holds: a gate/up tile has 16 gate rows and the
    // 16 up rows of the same outputs in every lane quarter
    const int erow = p.glu ? (lane & 15) + 16 * q + (lane >> 4) * 64 : q * 32 + lane;
    const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
    const uint32_t a_base = lane_base + kA0 + 32u * c2;

    // ---- epilogue of a job: this warp's NT / 4 tokens of its 32 lanes --------------------------
    auto epilogue = [&](int j) {
      const QmJob job = qm_job(p.deal, j);
      ok = ok && tc_wait_w(acc_full, (uint32_t)(j & 1), p.status);
      tc_after_sync();
      int si = 0;
      if (!p.glu) {
#pragma unroll
        for (int i = 1; i < kQmMaxSeg; ++i)
          if (i < p.nseg && job.tile >= p.seg[i].tile0) si = i;
      }
      const QmSeg& sg = p.seg[si];
      const int row = p.glu ? job.tile * 64 + 16 * q + (lane & 15)
                            : (job.tile - sg.tile0) * kQmRows + q * 32 + lane;
      const bool row_ok = ok && row < sg.N;
      // the whole share into registers, then the accumulator is free for the next job
      uint32_t va[NT / 64][16];
#pragma unroll
      for (int g = 0; g < NT / 64; ++g) {  // 16 tokens at a time
        uint32_t(&v)[16] = va[g];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
              "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
              "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(lane_base + (uint32_t)((warp >> 2) * (NT / 4) + 16 * g)));
      }
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      tc_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_free);
#pragma unroll
      for (int g = 0; g < NT / 64; ++g) {
        const int m0 = (warp >> 2) * (NT / 4) + 16 * g;
        if (m0 >= p.M) break;  // the same for the whole warp
        uint32_t(&v)[16] = va[g];
        if (job.slot >= 0) {
          // a part of a tile: four tokens of a row per 16-byte store
          float4* dst = reinterpret_cast<float4*>(p.part) +
                        (((size_t)blockIdx.x * 2 + job.slot) * (NT / 4) + (m0 >> 2)) * kQmRows + q * 32 + lane;
#pragma unroll
          for (int t = 0; t < 4; ++t)
            dst[t * kQmRows] = make_float4(__uint_as_float(v[4 * t]), __uint_as_float(v[4 * t + 1]),
                                           __uint_as_float(v[4 * t + 2]), __uint_as_float(v[4 * t + 3]));
          continue;
        }
        const int mc = min(16, p.M - m0);
        if (!p.glu) {
          const size_t o0 = (size_t)m0 * sg.ldy + row;
          if (row_ok) {
            float res[16];
            if (sg.residual) {
#pragma unroll
              for (int t = 0; t < 16; ++t) res[t] = t < mc ? sg.residual[o0 + (size_t)t * sg.ldy] : 0.f;
            }
#pragma unroll
            for (int t = 0; t < 16; ++t)
              if (t < mc) {
                const float r = __uint_as_float(v[t]) * rs_s[m0 + t];
                sg.y[o0 + (size_t)t * sg.ldy] = sg.residual ? __fadd_rn(r, res[t]) : r;
              }
          }
        } else {
          // gate lanes finish the even tokens, up lanes the odd ones
          const bool up = lane >= 16;
#pragma unroll
          for (int t = 0; t < 16; t += 2) {
            const float a = __uint_as_float(v[t]) * rs_s[m0 + t];
            const float b = __uint_as_float(v[t + 1]) * rs_s[m0 + t + 1];
            const float got = __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
            const float r = up ? glu_gate(got) * b : glu_gate(a) * got;
            const int tt = up ? t + 1 : t;
            if (row_ok && tt < mc) sg.y[(size_t)(m0 + tt) * sg.ldy + row] = r;
          }
        }
      }
    };

    bool waited = false;
    // the epilogue reads what the previous kernel wrote (row scales, residual)
    auto wait_previous = [&]() {
      if (waited) return;
      waited = true;
      pdl_wait();
      // this warp's tokens (the four warps that share them write the same values)
      for (int t = lane; t < NT / 4; t += 32) {
        const int m = (warp >> 2) * (NT / 4) + t;
        rs_s[m] = m < p.M ? __ldcg(p.rowscale + m) : 0.f;
      }
      __syncwarp();
    };
    if constexpr (Cfg::kSums) {  // the upper half of every residue slot meets zero columns: keep it finite
      if (warp < 4) {
#pragma unroll
        for (int e = 0; e < Cfg::kESlots; ++e)
          asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%1,%1,%1};" ::"r"(
                           lane_base + (uint32_t)(Cfg::kE0 + 8 * e + 4)), "r"(0)
                       : "memory");
      }
    }
    const bool epi = warp < kEpiWarps;
    int s = grp;       // this warp's stages: grp, grp + kGroups, ...
    int end = 0;       // first stage of the next job
    int pending = -1;  // job whose epilogue is due
    TcRing<kPkStages> rp;
    TcRing<kAStages> ra;
    rp.advance(grp / kAParts);
    ra.advance(grp);
    for (int j = 0; j < njobs; ++j) {
      end += kAParts * qm_job(p.deal, j).n;
      int since = 0;
      for (; s < end; s += kGroups) {
        ok = ok && tc_wait_w(&pk_full[rp.i], rp.phase, p.status);
        const uint8_t* blk = pk + (size_t)rp.i * kPkBytes + (size_t)erow * kUnit;
        const uint32_t a_t = a_base + ra.i * kACols;
        auto stage_free = [&]() {
          if (s >= kAStages) wait_previous();  // freed by a product, which needs the activations
          ok = ok && tc_wait_w(&a_free[ra.i], ra.phase ^ 1, p.status);
          tc_after_sync();
        };
        auto store16 = [&](uint32_t col, const uint32_t (&o)[16]) {
          asm volatile(
              "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
              "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(a_t + col),
              "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]),
              "r"(o[8]), "r"(o[9]), "r"(o[10]), "r"(o[11]), "r"(o[12]), "r"(o[13]), "r"(o[14]),
              "r"(o[15])
              : "memory");
        };
        uint4 hdr;
        bool wide = false;  // a row of this warp whose dmin * 63 f16 does not hold
        if constexpr (FMT == 12) {
          hdr = *reinterpret_cast<const uint4*>(blk);
          wide = __any_sync(0xffffffffu, (hdr.x & 0x7FFF0000u) > 0x640F0000u);  // |dmin| > 1039
        }
#pragma unroll
        for (int hh = 0; hh < 2 / kAParts; ++hh) {
          const int half = kAParts == 1 ? hh : (s & 1);
          const int c = 2 * half + c2;  // sub-blocks 2c, 2c+1
          const uint32_t col0 = 64u * hh;
          if constexpr (FMT == 12) {
            // super-block of this row: f16 d, f16 dmin, 12 bytes of 6-bit scales and mins, 128 bytes
            // of nibbles (Hesper/Quantization/Q4_K_M.lean:13-52,120-144)
            const uint4 qa = *reinterpret_cast<const uint4*>(blk + 16 + 32 * c);
            const uint4 qb = *reinterpret_cast<const uint4*>(blk + 32 + 32 * c);
            // scale / min bytes j and j+1 (j = 2c) out of the 12 packed bytes hdr.y, hdr.z, hdr.w
            uint32_t sc2, m2;  // two 6-bit values each, in bytes 0 and 1
            const int sh = 16 * c2;
            if (half == 0) {
              sc2 = (hdr.y >> sh) & 0x3F3Fu;
              m2 = (hdr.z >> sh) & 0x3F3Fu;
            } else {
              sc2 = ((hdr.w >> sh) & 0x0F0Fu) | ((hdr.y >> (sh + 2)) & 0x3030u);
              m2 = ((hdr.w >> (sh + 4)) & 0x0F0Fu) | ((hdr.z >> (sh + 2)) & 0x3030u);
            }
            // {scale 2c, scale 2c+1} as f16, then multiplier and addend of the two nibble positions
            const __half2 k1024 = __floats2half2_rn(1024.f, 1024.f);
            const __half2 sc = __hsub2(as_h2(__byte_perm(sc2, 0x64646464u, 0x4140)), k1024);
            const __half2 mn = __hsub2(as_h2(__byte_perm(m2, 0x64646464u, 0x4140)), k1024);
            const __half2 mul = __hmul2(sc, __floats2half2_rn(1.f, 0.0625f));
            const __half2 add = __hmul2(sc, __floats2half2_rn(-1024.f, -64.f));
            // c = -dmin * m rounded to f16, and 32 times what that lost (an f16 fma forms dmin * m + c
            // exactly up to its own rounding)
            const __half2 dm = __high2half2(as_h2(hdr.x));
            const __half2 cc = __hneg2(__hmul2(dm, mn));
            __half2 lost = __hmul2(__hfma2(dm, mn, cc), __floats2half2_rn(-32.f, -32.f));
            const uint32_t qq[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
            const __half2 d = __low2half2(as_h2(hdr.x));
            uint32_t o[16];
            q4k_expand<false>(qq, d, __low2half2(mul), __low2half2(add), __low2half2(cc), o);
            if (wide) {
              const float dm32 = -__high2float(as_h2(hdr.x));
              q4k_expand_f32<false>(qq, __low2float(d) * (float)(sc2 & 63u), dm32 * (float)(m2 & 63u), o);
              lost = __floats2half2_rn(0.f, 0.f);
            }
            if (hh == 0) stage_free();
            store16(col0, o);
            asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(
                             lane_base + (uint32_t)(Cfg::kE0 + 8 * ((s / kAParts) % Cfg::kESlots) + c)),
                         "r"(as_u32(lost))
                         : "memory");
            q4k_expand<true>(qq, d, __high2half2(mul), __high2half2(add), __high2half2(cc), o);
            if (wide) {
              const float dm32 = -__high2float(as_h2(hdr.x));
              q4k_expand_f32<true>(qq, __low2float(d) * (float)(sc2 >> 8), dm32 * (float)(m2 >> 8), o);
            }
            store16(col0 + 16, o);
          } else {
            // Q8_0 (Hesper/Layers/Linear.lean:6207-6223): blocks 2c and 2c+1 of the row's eight, 34
            // bytes each -- f16 d, then 32 int8.  The chunk starts on a word; block 2c's quants sit
            // two bytes into it (funnel shifts), block 2c+1's are word aligned.
            const uint32_t* wq = reinterpret_cast<const uint32_t*>(blk + 68 * c);
            uint32_t w[9], o[16];
#pragma unroll
            for (int i = 0; i < 9; ++i) w[i] = wq[i];
            const __half2 d0 = __half2half2(__ushort_as_half((unsigned short)(w[0] & 0xFFFFu)));
            const __half2 d1 = __half2half2(__ushort_as_half((unsigned short)(w[8] >> 16)));
#pragma unroll
            for (int i = 0; i < 8; ++i)
              q80_word(__funnelshift_r(w[i], w[i + 1], 16), d0, o[2 * i], o[2 * i + 1]);
            if (hh == 0) stage_free();
            store16(col0, o);
#pragma unroll
            for (int i = 0; i < 8; ++i) q80_word(wq[9 + i], d1, o[2 * i], o[2 * i + 1]);
            store16(col0 + 16, o);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&pk_free[rp.i]);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&a_full[ra.i]);
        ra.advance(kGroups);
        rp.advance(kAParts == 1 ? kGroups : ((s & 1) + kGroups) >> 1);
        // the A stages are refilled for this job: now the previous job's accumulator
        if (pending >= 0 && ++since == kAStages / kGroups) {
          wait_previous();
          epilogue(pending);
          pending = -1;
        }
      }
      if (pending >= 0) {
        wait_previous();
        epilogue(pending);
      }
      pending = epi ? j : -1;
    }
    wait_previous();
    if (pending >= 0) epilogue(pending);
  }
  tc_before_sync();
  __syncthreads();
  if (warp == kMmaWarp)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(*tmem_slot));
}

// Adds the partials of the left-over tiles in K order and runs the epilogue on the sums: a thread
// per tensor-memory lane and four tokens.
__global__ void __launch_bounds__(128) kq_combine_kernel(const __grid_constant__ QmParams p, int NT,
                                                         int grid) {
  pdl_trigger();
  pdl_wait();
  const int l = threadIdx.x, m0 = blockIdx.y * 4;
  const int t = blockIdx.x, nb = p.deal.nb, upc = p.deal.upc;
  const int c0 = t * nb / upc, c1 = ((t + 1) * nb - 1) / upc;
  if (c0 == c1) return;  // one CTA did the whole tile and has stored it
  const float4* part = reinterpret_cast<const float4*>(p.part) + (size_t)(m0 >> 2) * kQmRows + l;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int cb = c0; cb <= c1; cb += 8) {  // eight partials in flight
    float4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int cta = cb + i, slot = t - cta * upc / nb;
      v[i] = cta <= c1 ? __ldcg(part + ((size_t)cta * 2 + slot) * (NT / 4) * kQmRows)
                       : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      a.x = __fadd_rn(a.x, v[i].x); a.y = __fadd_rn(a.y, v[i].y);
      a.z = __fadd_rn(a.z, v[i].z); a.w = __fadd_rn(a.w, v[i].w);
    }
  }
  const float4 rs = __ldcg(reinterpret_cast<const float4*>(p.rowscale + m0));
  const float r[4] = {a.x * rs.x, a.y * rs.y, a.z * rs.z, a.w * rs.w};
  const int tile = p.deal.W * grid + t, mc = min(4, p.M - m0);
  if (!p.glu) {
    int si = 0;
#pragma unroll
    for (int i = 1; i < kQmMaxSeg; ++i)
      if (i < p.nseg && tile >= p.seg[i].tile0) si = i;
    const QmSeg& sg = p.seg[si];
    const int row = (tile - sg.tile0) * kQmRows + l;
    const size_t o = (size_t)m0 * sg.ldy + row;
    if (row < sg.N) {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (e < mc) {
          const size_t i = o + (size_t)e * sg.ldy;
          sg.y[i] = sg.residual ? __fadd_rn(r[e], sg.residual[i]) : r[e];
        }
    }
  } else {  // lanes 32q..32q+15 hold gate rows, lanes 32q+16..32q+31 their up rows
    const QmSeg& sg = p.seg[0];
    const bool up = l & 16;
    const int row = tile * 64 + 16 * (l >> 5) + (l & 15);
#pragma unroll
    for (int e = 0; e < 4; e += 2) {  // gate lanes finish the even tokens, up lanes the odd ones
      const float got = __shfl_xor_sync(0xffffffffu, up ? r[e] : r[e + 1], 16);
      const float y = up ? glu_gate(got) * r[e + 1] : glu_gate(r[e]) * got;
      const int ee = up ? e + 1 : e;
      if (row < sg.N && ee < mc) sg.y[(size_t)(m0 + ee) * sg.ldy + row] = y;
    }
  }
}

}  // namespace hb

using namespace hb;

// Dealing `tiles` row tiles of `nb` super-blocks to the SMs: whole waves, then the rest cut into
// equal runs of units.  The rest stays whole (upc = nb) when cutting it saves less than the
// partials cost: a unit takes a CTA about max(800, 16 * (NT / 2 + 10)) cycles, partials and the
// second kernel about 4000 + 12 NT.
static QmDeal qm_deal(int tiles, int nb, int NT, int sms, int* grid) {
  QmDeal d = {tiles / sms, tiles % sms, nb, nb};
  if (d.R) {
    const int upc = (d.R * nb + sms - 1) / sms;
    const int unit = 16 * (NT / 2 + 10) > 800 ? 16 * (NT / 2 + 10) : 800;
    if ((long)(nb - upc) * unit > 4000 + 12 * NT) d.upc = upc;
  }
  *grid = d.W ? sms : (d.R * nb + d.upc - 1) / d.upc;
  return d;
}

template <int NT, int FMT>
static int kq_mma_launch(hb200_ctx* ctx, QmParams& p, int tiles, int nb, cudaStream_t st) {
  using Cfg = QmCfg<NT, FMT>;
  int grid = 0;
  p.deal = qm_deal(tiles, nb, NT, ctx->sm_count, &grid);
  if (p.deal.upc < nb &&
      (size_t)grid * 2 * NT * kQmRows * sizeof(float) > kScratchBytes - kScratchSplitK) {
    p.deal.upc = nb;  // more SMs than the partials' region was laid out for
    grid = p.deal.W ? ctx->sm_count : p.deal.R;
  }
  const int rc = hb_func_smem(ctx, reinterpret_cast<const void*>(kq_mma_kernel<NT, FMT>),
                              (size_t)Cfg::kSmem);
  if (rc != HB200_OK) return rc;
  HB_CUDA(launch_pdl(kq_mma_kernel<NT, FMT>, dim3((unsigned)grid), dim3(Cfg::kThreads),
                     (size_t)Cfg::kSmem, st, ctx->pdl, p));
  if (p.deal.R && p.deal.upc < nb)
    HB_CUDA(launch_pdl(kq_combine_kernel, dim3((unsigned)p.deal.R, (unsigned)((p.M + 3) / 4)), dim3(128),
                       0, st, ctx->pdl, p, NT, grid));
  return HB200_OK;
}

// For each of nseg tensors: y[m*ldy + n] = sum_k dequant(W)[n,k] x[m,k] (+ residual) for the
// M <= NT tokens staged by hb_kq_stage for the same NT (64, 128 or 256) and format, all in ONE
// product launch.  glu != 0: two tensors of equal shape, gate and
// up, and segs[0].y = gelu_tanh(gate) * up.  Q4_K or Q8_0 (fmt: the GGUF type id); K a multiple
// of 256.
int hb_kq_mma_run_multi(hb200_ctx* ctx, const HbKqSeg* segs, int nseg, int K, int M, int NT, int glu,
                        cudaStream_t st, int fmt) {
  HB_REQUIRE(fmt == HB200_FMT_Q4_K || fmt == HB200_FMT_Q8_0, "kquant (fused batched): format %d", fmt);
  HB_REQUIRE(nseg >= 1 && nseg <= kQmMaxSeg && K % 256 == 0 && M >= 1 && M <= NT &&
                 (NT == 64 || NT == 128 || NT == 256) && (!glu || (nseg == 2 && segs[0].N == segs[1].N)),
             "kquant (fused batched): nseg=%d K=%d M=%d NT=%d", nseg, K, M, NT);
  QmParams p = {};
  TcEncodeTiledFn encode = tc_tensor_map_encoder();
  HB_REQUIRE(encode != nullptr, "kquant (fused batched): the driver has no cuTensorMapEncodeTiled");
  const int unit = fmt == HB200_FMT_Q4_K ? 144 : 272;  // bytes of 256 weights
  const int rowbytes = K / 256 * unit;
  int tiles = 0;
  for (int s = 0; s < nseg; ++s) {
    const HbKqSeg& g = segs[s];
    HB_REQUIRE(g.N >= 1 && g.N < (1l << 31) && g.blocks && g.y,
               "kquant (fused batched): tensor %d has no rows or a null pointer", s);
    // Q4_K: bytes; Q8_0: 32-bit words (a box dimension holds at most 256 elements, 272 > 256)
    const int esz = fmt == HB200_FMT_Q4_K ? 1 : 4;
    const cuuint64_t dims[2] = {(cuuint64_t)(rowbytes / esz), (cuuint64_t)g.N};
    const cuuint64_t strides[1] = {(cuuint64_t)rowbytes};
    const cuuint32_t box[2] = {(cuuint32_t)(unit / esz), (cuuint32_t)(kQmRows / 2)};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult rc = encode(&p.tmap[s],
                               esz == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_UINT32, 2,
                               const_cast<uint8_t*>(g.blocks), dims, strides, box, estr,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    HB_REQUIRE(rc == CUDA_SUCCESS, "kquant (fused batched): cuTensorMapEncodeTiled failed (%d)",
               (int)rc);
    p.seg[s] = {g.residual, g.y, g.ldy, (int)g.N, tiles};
    if (!glu) tiles += (int)((g.N + kQmRows - 1) / kQmRows);
  }
  if (glu) tiles = (int)((segs[0].N + kQmRows / 2 - 1) / (kQmRows / 2));
  p.nseg = nseg;
  p.glu = glu;
  p.xb = static_cast<const uint8_t*>(ctx->d_scratch) + kScratchKqActs;
  p.rowscale = reinterpret_cast<const float*>(static_cast<const uint8_t*>(ctx->d_scratch) +
                                              kScratchRowScale);
  p.M = M;
  p.part = reinterpret_cast<float*>(static_cast<uint8_t*>(ctx->d_scratch) + kScratchSplitK);
  p.status = ctx->d_status;
  const int nb = K / 256;
  if (fmt == HB200_FMT_Q4_K) {
    switch (NT) {
      case 64: return kq_mma_launch<64, 12>(ctx, p, tiles, nb, st);
      case 128: return kq_mma_launch<128, 12>(ctx, p, tiles, nb, st);
      default: return kq_mma_launch<256, 12>(ctx, p, tiles, nb, st);
    }
  }
  switch (NT) {
    case 64: return kq_mma_launch<64, 8>(ctx, p, tiles, nb, st);
    case 128: return kq_mma_launch<128, 8>(ctx, p, tiles, nb, st);
    default: return kq_mma_launch<256, 8>(ctx, p, tiles, nb, st);
  }
}

// Bytes of staged activations per super-block of 256 weights.
static size_t qm_sb_bytes(int fmt, int NT) { return (size_t)NT * (fmt == HB200_FMT_Q4_K ? 544 : 512); }

constexpr size_t kQmActBytes = kScratchRowScale - kScratchKqActs;
constexpr int kQmMaxK = 65280;
static_assert((size_t)64 * 544 * (kQmMaxK / 256) <= kQmActBytes, "a pass of 64 tokens fits at every K");

// Most tokens (64, 128 or 256) one pass can stage at this K.
int hb_kq_mma_max_tokens(int fmt, int K) {
  for (int NT = 256; NT > 64; NT >>= 1)
    if (qm_sb_bytes(fmt, NT) * (size_t)(K / 256) <= kQmActBytes) return NT;
  return 64;
}

template <bool I8>
static int qm_stage_launch(hb200_ctx* ctx, const QmStage& p, int rows, cudaStream_t st) {
  const int n8 = p.K / 8;  // groups of 8 elements; one or two per thread, eight for a huge row
  const int G = n8 <= 640 ? 1 : (n8 <= 2048 ? 2 : 8);
  const int threads = ((n8 + G - 1) / G + 31) & ~31;
  auto kern = G == 1 ? kq_stage_kernel<1, I8> : (G == 2 ? kq_stage_kernel<2, I8> : kq_stage_kernel<8, I8>);
  HB_CUDA(launch_pdl(kern, dim3(rows), dim3(threads), 0, st, ctx->pdl, p));
  return HB200_OK;
}

// x[M][K] (M <= NT) -> f16 operand layout and row scales in the context scratch; optional pre-step
// x' = d_pre_base + rmsnorm(d_x) * d_pre_gamma (written to d_pre_out), optional RMSNorm.
int hb_kq_stage(hb200_ctx* ctx, int fmt, int K, int NT, const float* d_x, int M,
                const float* d_pre_base, const float* d_pre_gamma, float* d_pre_out,
                const float* d_rms_gamma, float rms_eps, cudaStream_t st) {
  QmStage p = {};
  p.sb_bytes = qm_sb_bytes(fmt, NT);
  p.sums_off = fmt == HB200_FMT_Q4_K ? NT * 512 : 0;
  HB_REQUIRE(p.sb_bytes * (size_t)(K / 256) <= kQmActBytes && K <= kQmMaxK,
             "kquant (fused batched): K=%d does not fit the activation scratch", K);
  p.x = d_x;
  p.gamma = d_rms_gamma;
  p.pre_base = d_pre_base;
  p.pre_gamma = d_pre_gamma;
  p.pre_out = d_pre_out;
  p.eps = rms_eps;
  p.K = K;
  p.xb = static_cast<uint8_t*>(ctx->d_scratch) + kScratchKqActs;
  p.rowscale = reinterpret_cast<float*>(static_cast<uint8_t*>(ctx->d_scratch) + kScratchRowScale);
  return qm_stage_launch<false>(ctx, p, M, st);
}

// The same for the few-token kernel (kquant_sb.cu), into `frag`: ntl * 8 token columns, M of them real.
int hb_kq_stage_i8(hb200_ctx* ctx, int fmt, int K, int ntl, const float* d_x, int M, const float* d_pre_base,
                   const float* d_pre_gamma, float* d_pre_out, const float* d_rms_gamma, float rms_eps,
                   uint8_t* frag, cudaStream_t st) {
  QmStage p = {};
  p.sb_bytes = (size_t)ntl * 4608;
  p.sums_off = fmt == HB200_FMT_Q4_K;
  HB_REQUIRE(K <= 65536, "kquant (few tokens): K=%d", K);
  p.x = d_x;
  p.gamma = d_rms_gamma;
  p.pre_base = d_pre_base;
  p.pre_gamma = d_pre_gamma;
  p.pre_out = d_pre_out;
  p.eps = rms_eps;
  p.K = K;
  p.M = M;
  p.ntl = ntl;
  p.xb = frag;
  return qm_stage_launch<true>(ctx, p, ntl * 8, st);
}
