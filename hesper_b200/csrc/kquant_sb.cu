// kquant_sb.cu -- Q4_K / Q8_0 product for a handful of tokens (2 to 15) on the integer tensor-core
// instruction.
//
// Same contract and the same arithmetic as the streaming kernel of kquant.cu (the reference's
// counterparts are the M>1 paths of Hesper/Layers/Linear.lean:1152-1760,5973-6177): activations in
// 16 bits per 32 elements, x ~ dx * (256*hi + lo), exact integer products, f32 scales and sums.  The
// streaming kernel repeats its dp4a loop and its weight stream once per token (Q8_0 K=2560
// N=10240: 36.9 us at 7 tokens, 11.7 here); here the weights are read once and the tokens are the columns of
// mma.sync.m16n8k32, so a few tokens cost about what one does.  f16 operands (the tcgen05
// path from 16 tokens on) would round weights and activations to 2^-11; these do not.
//
//   * staging (kq_stage_kernel in kquant_mma.cu, one CTA per token): norm, 16-bit quantisation, and
//     the B fragments as a lane wants them: per 32 elements and 8 tokens 32 lanes x {hi, hi, lo, lo};
//   * product: the rows of every tensor are dealt evenly to the CTAs (to the row, not to the tile: a
//     tile's missing rows repeat its last one).  A CTA walks its rows in passes of at most 128 and
//     each pass along K; a pipeline stage is one super-block (256 weights) of the pass's rows -- one
//     tensor-map box, plus a second one for the up rows of a gate/up pair -- and its fragments.
//     The weights of the first stages are fetched before griddepcontrol.wait, under the staging
//     kernel.  16 warps: one per 16-row tile and K group (warp = kg * tiles + tile, K group kg
//     takes the positions kg, kg + KG, ... of the CTA's walk); the K groups meet in shared memory in
//     fixed order.
//     A parity wait tells a slot's lap from the next one only, so whoever waits for a lap has to
//     know that the one before has landed: every slot belongs to one K group (the ring's stages are
//     a multiple of KG, the position decides the group), or the ring never wraps (sb_plan).
//
// What bounds it is latency, not a rate: at K=2560 N=10240 instruction issue takes 2 to 3.5 us (about 330
// instructions per 16 rows x 256 weights at up to 8 tokens, 520 at up to 15) and the weight stream
// 2.3 (Q4_K) or 4.3 us (Q8_0), the call 9 to 12: the staging launch (2 to 3), a CTA's fill and, per pass,
// the chain from a stage's arrival through two dependent products per 32 weights and token column.
#include <optional>
#include <type_traits>

#include "tcgen05.cuh"

namespace hb {

constexpr int kSbWarps = 16;                      // consumer warps; one more copies
constexpr int kSbThreads = (kSbWarps + 1) * 32;
constexpr int kSbMaxSeg = 4;
constexpr int kSbRows = 128;                      // most MMA rows of a pass
constexpr int kSbMaxStages = 32;
constexpr int kSbCtrl = 1024;

struct SbSeg {
  const float* residual;  // nullable
  float* y;
  int N;
  int cta0, ctas;  // CTAs [cta0, cta0 + ctas) own this tensor's rows
  int rp;          // rows of a pass (gate/up: outputs)
  int tiles;       // 16-row tiles of a pass
  int groups;      // K groups of warps
  int stages;      // stages of this tensor's ring
};

struct SbParams {
  CUtensorMap tmap[kSbMaxSeg];  // blocks as [N rows][rowbytes], boxes of rp rows x one super-block
  SbSeg seg[kSbMaxSeg];
  int nseg, gu;   // gu: segments 0 and 1 are gate and up; the result goes to segment 0's y
  int nsb, M;
  int wbytes;          // bytes of a stage before its fragments
  const uint8_t* xb;
  uint32_t* status;
};

template <int FMT, int NTL>  // NTL: token columns / 8
struct SbCfg {
  static constexpr int kUnit = FMT == 12 ? 144 : 272;
  static constexpr int kFrag = NTL * 4096;               // [8 sub-blocks][NTL][32 lanes][16]
  static constexpr int kB = kFrag + NTL * 512;           // + [8][NTL][4]{dx, dx, sum, sum}
  static constexpr int kPart = kSbWarps * NTL * 4 * 32 * 4;
};

template <bool SIGNED_A>
__device__ __forceinline__ void sb_mma(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (SIGNED_A)
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// d * (byte b of w) in f32, exact (d an f16, the byte at most 6 bits): the byte becomes the mantissa
// of 2^23 + byte, the fma takes d * 2^23 off again.
template <int B>
__device__ __forceinline__ float sb_scale(uint32_t w, float d, float d23) {
  return fmaf(d, __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540 | B)), -d23);
}

__device__ __forceinline__ float sb_gelu_tanh(float x) {
  // Hesper/Layers/FusedFFNSpec.lean:42-45
  const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  return 0.5f * x * (1.0f + tanhf(u));
}

// One sub-block J: products of 16 rows x 32 weights with NTL x 8 tokens, scaled into acc.
// acc[n][0..3]: (row g, token 8n+2t), (g, +1), (row g+8, ...), (g+8, +1).
template <int FMT, int NTL, int J>
__device__ __forceinline__ void sb_block(const uint32_t (&a)[4], const uint8_t* bst, int lane, float sA, float sB,
                                         float mA, float mB, float (&acc)[NTL][4]) {
  using Cfg = SbCfg<FMT, NTL>;
#pragma unroll
  for (int n = 0; n < NTL; ++n) {
    const uint4 bf = *reinterpret_cast<const uint4*>(bst + (J * NTL + n) * 512 + lane * 16);
    const float4 tb = *reinterpret_cast<const float4*>(bst + Cfg::kFrag + ((J * NTL + n) * 4 + (lane & 3)) * 16);
    int c[4] = {0, 0, 0, 0};
    sb_mma<FMT == 8>(c, a, bf.x, bf.y);
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] *= 256;
    sb_mma<FMT == 8>(c, a, bf.z, bf.w);
    acc[n][0] = fmaf(sA * (float)c[0], tb.x, acc[n][0]);
    acc[n][1] = fmaf(sA * (float)c[1], tb.y, acc[n][1]);
    acc[n][2] = fmaf(sB * (float)c[2], tb.x, acc[n][2]);
    acc[n][3] = fmaf(sB * (float)c[3], tb.y, acc[n][3]);
    if constexpr (FMT == 12) {
      acc[n][0] = fmaf(mA, tb.z, acc[n][0]);
      acc[n][1] = fmaf(mA, tb.w, acc[n][1]);
      acc[n][2] = fmaf(mB, tb.z, acc[n][2]);
      acc[n][3] = fmaf(mB, tb.w, acc[n][3]);
    }
  }
}

// One super-block of a tile: rA, rB = the super-block of the lane's rows g and g + 8.
template <int NTL>
__device__ __forceinline__ void sb_unit_q4k(const uint8_t* rA, const uint8_t* rB, const uint8_t* bst, int lane,
                                            float (&acc)[NTL][4]) {
  const int t = lane & 3;
  const uint4 hA = *reinterpret_cast<const uint4*>(rA), hB = *reinterpret_cast<const uint4*>(rB);
  const float2 ddA = __half22float2(*reinterpret_cast<const __half2*>(&hA.x));
  const float2 ddB = __half22float2(*reinterpret_cast<const __half2*>(&hB.x));
  const float dA23 = ddA.x * 8388608.f, dB23 = ddB.x * 8388608.f;
  const float nA = -ddA.y, nB = -ddB.y, nA23 = nA * 8388608.f, nB23 = nB * 8388608.f;
  // six-bit scales and mins of sub-blocks 0..3 and 4..7 (Hesper/Quantization/Q4_K_M.lean:120-144)
  auto lowq = [](uint32_t v) { return v & 0x3F3F3F3Fu; };
  auto highq = [](uint32_t w, uint32_t v) { return (w & 0x0F0F0F0Fu) | ((v >> 2) & 0x30303030u); };
  const uint32_t sA[2] = {lowq(hA.y), highq(hA.w, hA.y)}, sB[2] = {lowq(hB.y), highq(hB.w, hB.y)};
  const uint32_t mA[2] = {lowq(hA.z), highq(hA.w >> 4, hA.z)}, mB[2] = {lowq(hB.z), highq(hB.w >> 4, hB.z)};
  auto chunk = [&](auto cc) {  // sub-blocks 2c (low nibbles) and 2c+1 (high, in place: 16 q)
    constexpr int c = decltype(cc)::value, h = c >> 1, b = 2 * (c & 1);
    const uint2 wa = *reinterpret_cast<const uint2*>(rA + 16 + 32 * c + 8 * t);
    const uint2 wb = *reinterpret_cast<const uint2*>(rB + 16 + 32 * c + 8 * t);
    constexpr uint32_t L = 0x0F0F0F0Fu, H = 0xF0F0F0F0u;
    const uint32_t lo[4] = {wa.x & L, wb.x & L, wa.y & L, wb.y & L};
    const uint32_t hi[4] = {wa.x & H, wb.x & H, wa.y & H, wb.y & H};
    sb_block<12, NTL, 2 * c>(lo, bst, lane, sb_scale<b>(sA[h], ddA.x, dA23), sb_scale<b>(sB[h], ddB.x, dB23),
                             sb_scale<b>(mA[h], nA, nA23), sb_scale<b>(mB[h], nB, nB23), acc);
    sb_block<12, NTL, 2 * c + 1>(hi, bst, lane, sb_scale<b + 1>(sA[h], ddA.x, dA23),
                                 sb_scale<b + 1>(sB[h], ddB.x, dB23), sb_scale<b + 1>(mA[h], nA, nA23),
                                 sb_scale<b + 1>(mB[h], nB, nB23), acc);
  };
  chunk(std::integral_constant<int, 0>{});
  chunk(std::integral_constant<int, 1>{});
  chunk(std::integral_constant<int, 2>{});
  chunk(std::integral_constant<int, 3>{});
}

// Eight Q8_0 blocks of 34 bytes: f16 d, then 32 int8 (Hesper/Layers/Linear.lean:6207-6223).  Even
// blocks' quants sit two bytes into a word (funnel shifts), odd blocks' are word aligned.
template <int NTL>
__device__ __forceinline__ void sb_unit_q80(const uint8_t* rA, const uint8_t* rB, const uint8_t* bst, int lane,
                                            float (&acc)[NTL][4]) {
  const int t = lane & 3;
  auto half_at = [](const uint8_t* p) { return __half2float(*reinterpret_cast<const __half*>(p)); };
  auto chunk = [&](auto cc) {
    constexpr int c = decltype(cc)::value;
    const uint32_t* ea = reinterpret_cast<const uint32_t*>(rA + 68 * c + 8 * t);
    const uint32_t* eb = reinterpret_cast<const uint32_t*>(rB + 68 * c + 8 * t);
    const uint32_t a0 = ea[0], a1 = ea[1], a2 = ea[2], b0 = eb[0], b1 = eb[1], b2 = eb[2];
    const uint32_t ev[4] = {__funnelshift_r(a0, a1, 16), __funnelshift_r(b0, b1, 16), __funnelshift_r(a1, a2, 16),
                            __funnelshift_r(b1, b2, 16)};
    sb_block<8, NTL, 2 * c>(ev, bst, lane, half_at(rA + 68 * c), half_at(rB + 68 * c), 0.f, 0.f, acc);
    const uint32_t od[4] = {ea[9], eb[9], ea[10], eb[10]};
    sb_block<8, NTL, 2 * c + 1>(od, bst, lane, half_at(rA + 68 * c + 34), half_at(rB + 68 * c + 34), 0.f, 0.f, acc);
  };
  chunk(std::integral_constant<int, 0>{});
  chunk(std::integral_constant<int, 1>{});
  chunk(std::integral_constant<int, 2>{});
  chunk(std::integral_constant<int, 3>{});
}

template <int FMT, int NTL>
__global__ void __launch_bounds__(kSbThreads, 1) kq_sb_kernel(const __grid_constant__ SbParams p) {
  using Cfg = SbCfg<FMT, NTL>;
  constexpr int kUnit = Cfg::kUnit;
  constexpr int kBoxX = FMT == 12 ? 144 : 68;  // map elements of a super-block: bytes, words
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);  // [stages] weights and fragments landed
  uint64_t* empty = full + kSbMaxStages;               // [stages] the tile warps have read it
  float* part = reinterpret_cast<float*>(smem + kSbCtrl);
  uint8_t* ring = smem + kSbCtrl + Cfg::kPart;
  const int nsb = p.nsb;
  const size_t stage_bytes = (size_t)p.wbytes + Cfg::kB;

  int si = 0;
  if (!p.gu) {
#pragma unroll
    for (int s = 1; s < kSbMaxSeg; ++s)
      if (s < p.nseg && (int)blockIdx.x >= p.seg[s].cta0) si = s;
  }
  const SbSeg& sg = p.seg[si];
  const int ci = (int)blockIdx.x - sg.cta0, rp = sg.rp, tiles = sg.tiles, S = sg.stages;
  const int r0 = (int)((long long)sg.N * ci / sg.ctas), r1 = (int)((long long)sg.N * (ci + 1) / sg.ctas);
  const int npass = (r1 - r0 + rp - 1) / rp;
  const int boxbytes = rp * kUnit, up_off = (boxbytes + 127) & ~127;

  if (tid == 0) {
    for (int i = 0; i < S; ++i) {
      mbar_init(&full[i], 2);  // one arrival with the weight bytes, one with the fragments
      mbar_init(&empty[i], tiles);
    }
    fence_mbar_init();
  }
  __syncthreads();
  pdl_trigger();

  if (warp == kSbWarps) {
    // ================= copies ====================================================================
    if (lane == 0) {
      const uint64_t pol = policy_evict_first();
      const int total = npass * nsb;
      const uint32_t wtx = (uint32_t)boxbytes * (p.gu ? 2u : 1u);
      auto weights = [&](int st, int row, int sb) {
        uint8_t* dst = ring + (size_t)st * stage_bytes;
        mbar_arrive_expect_tx(&full[st], wtx);
        tc_tma_box_2d(dst, &p.tmap[si], sb * kBoxX, row, &full[st], pol);
        if (p.gu) tc_tma_box_2d(dst + up_off, &p.tmap[1], sb * kBoxX, row, &full[st], pol);
      };
      auto fragments = [&](int st, int sb) {
        mbar_arrive_expect_tx(&full[st], Cfg::kB);
        bulk_g2s(ring + (size_t)st * stage_bytes + p.wbytes, p.xb + (size_t)sb * Cfg::kB, Cfg::kB, &full[st]);
      };
      const int pre = min(S, total);
      for (int i = 0, sb = 0, row = r0; i < pre; ++i) {  // constants: no wait on the previous kernel
        weights(i, row, sb);
        if (++sb == nsb) sb = 0, row += rp;
      }
      pdl_wait();  // the fragments come from the kernel before this one
      bool ok = true;
      int st = 0, sb = 0, row = r0;
      uint32_t phase = 1;
      for (int i = 0; i < total && ok; ++i) {
        if (i >= S) {
          ok = tc_wait(true, &empty[st], phase, p.status);
          if (!ok) break;
          weights(st, row, sb);
        }
        fragments(st, sb);
        if (++sb == nsb) sb = 0, row += rp;
        if (++st == S) st = 0, phase ^= 1;
      }
    }
  } else {
    // ================= products ===================================================================
    const int KG = sg.groups;
    const int tile = warp % tiles, kg = warp / tiles;
    const bool active = kg < KG;
    const int g = lane >> 2, t = lane & 3;
    bool ok = true;
    pdl_wait();  // the fragments and the residual; the output may still be read before this
    for (int ps = 0; ps < npass; ++ps) {
      const int row = r0 + ps * rp, nrows = min(rp, r1 - row);
      float acc[NTL][4];
#pragma unroll
      for (int n = 0; n < NTL; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
      if (active) {
        // rows past the pass's last one repeat it; their results are dropped
        const int ra = p.gu ? min(8 * tile + g, nrows - 1) : min(16 * tile + g, nrows - 1);
        const int rb = p.gu ? ra : min(16 * tile + g + 8, nrows - 1);
        const size_t oa = (size_t)ra * kUnit, ob = (size_t)rb * kUnit + (p.gu ? up_off : 0);
        // first position of this pass that is this group's: pos % KG == kg
        const int pos0 = ps * nsb, end = pos0 + nsb;
        for (int pos = pos0 + (kg - pos0 % KG + KG) % KG; pos < end; pos += KG) {
          const int lap = pos / S, st = pos - lap * S;
          ok = tc_wait(ok, &full[st], (uint32_t)(lap & 1), p.status);
          const uint8_t* w = ring + (size_t)st * stage_bytes;
          if constexpr (FMT == 12) sb_unit_q4k<NTL>(w + oa, w + ob, w + p.wbytes, lane, acc);
          else sb_unit_q80<NTL>(w + oa, w + ob, w + p.wbytes, lane, acc);
          __syncwarp();
          if (lane == 0) mbar_arrive(&empty[st]);
        }
      }
      // the K groups of a tile meet in shared memory, in order
      if (active && kg > 0) {
#pragma unroll
        for (int n = 0; n < NTL; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i) part[((warp * NTL + n) * 4 + i) * 32 + lane] = acc[n][i];
      }
      asm volatile("bar.sync 1, %0;" ::"n"(kSbWarps * 32) : "memory");
      if (kg == 0) {
        for (int k = 1; k < KG; ++k)
#pragma unroll
          for (int n = 0; n < NTL; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[n][i] += part[(((k * tiles + tile) * NTL + n) * 4 + i) * 32 + lane];
      }
      if (ps + 1 < npass) asm volatile("bar.sync 1, %0;" ::"n"(kSbWarps * 32) : "memory");
      if (kg != 0 || !ok) continue;
#pragma unroll
      for (int n = 0; n < NTL; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int m = 8 * n + 2 * t + e;
          if (m >= p.M) continue;
          if (p.gu) {
            if (8 * tile + g < nrows)
              sg.y[(size_t)m * sg.N + row + 8 * tile + g] = sb_gelu_tanh(acc[n][e]) * acc[n][2 + e];
          } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int lr = 16 * tile + g + 8 * h;
              if (lr >= nrows) continue;
              const size_t o = (size_t)m * sg.N + row + lr;
              float v = acc[n][2 * h + e];
              if (sg.residual) v += __ldcg(sg.residual + o);
              sg.y[o] = v;
            }
          }
        }
    }
  }
}

}  // namespace hb

using namespace hb;

// How the rows are dealt and how deep each tensor's ring is: host arithmetic only.
struct SbPlan {
  int grid, wbytes;    // bytes of a stage before its fragments, the same for every tensor
  size_t smem;
  int ctas[kSbMaxSeg], rp[kSbMaxSeg], tiles[kSbMaxSeg], groups[kSbMaxSeg], stages[kSbMaxSeg];
  int total[kSbMaxSeg];  // positions of the longest walk: passes x super-blocks
};

// N: rows of the tensors (gu: gate and up).  False: shape not covered.
static bool sb_plan(int fmt, int K, const int* N, int nseg, int gu, int M, int sms, int smem_optin, SbPlan* out) {
  if (M < 2 || M > 15 || K < 256 || K % 256 || K > 65536 || nseg < 1 || nseg > kSbMaxSeg || sms < nseg) return false;
  const int NTL = M <= 8 ? 1 : 2, nsb = K / 256;
  const int unit = fmt == HB200_FMT_Q4_K ? 144 : 272;
  const size_t bbytes = (size_t)NTL * (4096 + 512), part = (size_t)kSbWarps * NTL * 512;
  SbPlan p = {};
  const int work = gu ? 1 : nseg;  // tensors whose rows are dealt
  // CTAs per tensor: one each, then always to the one with the most rows per CTA, down to 4 rows
  for (int s = 0; s < work; ++s) p.ctas[s] = 1;
  p.grid = work;
  while (p.grid < sms) {
    int b = 0;
    for (int s = 1; s < work; ++s)
      if ((long long)N[s] * p.ctas[b] > (long long)N[b] * p.ctas[s]) b = s;
    if ((long long)N[b] <= 4ll * p.ctas[b]) break;
    ++p.ctas[b];
    ++p.grid;
  }
  const int cap = gu ? kSbRows / 2 : kSbRows;
  for (int s = 0; s < work; ++s) {
    const int most = (N[s] + p.ctas[s] - 1) / p.ctas[s], np = (most + cap - 1) / cap;
    p.rp[s] = (most + np - 1) / np;
    p.tiles[s] = gu ? (p.rp[s] + 7) / 8 : (p.rp[s] + 15) / 16;
    p.total[s] = np * nsb;
    const int wb = ((p.rp[s] * unit + 127) & ~127) * (gu ? 2 : 1);
    if (wb > p.wbytes) p.wbytes = wb;
  }
  if ((size_t)smem_optin < kSbCtrl + part) return false;
  const size_t stage = (size_t)p.wbytes + bbytes, fit = ((size_t)smem_optin - kSbCtrl - part) / stage;
  const int S = fit > (size_t)kSbMaxStages ? kSbMaxStages : (int)fit;
  if (S < 1) return false;
  int most = 1;
  for (int s = 0; s < work; ++s) {
    int g = kSbWarps / p.tiles[s];
    if (g > S) g = S;
    if (g > p.total[s]) g = p.total[s];
    p.groups[s] = g;
    // a ring that wraps holds a whole number of laps of the groups: each slot is one group's
    p.stages[s] = p.total[s] <= S ? p.total[s] : S - S % g;
    if (p.stages[s] > most) most = p.stages[s];
  }
  for (int s = work; s < nseg; ++s) {  // the up tensor goes with the gate
    p.ctas[s] = p.ctas[0], p.rp[s] = p.rp[0], p.tiles[s] = p.tiles[0];
    p.groups[s] = p.groups[0], p.stages[s] = p.stages[0], p.total[s] = p.total[0];
  }
  p.smem = kSbCtrl + part + (size_t)most * stage;
  *out = p;
  return true;
}

extern "C" int hb200_kquant_few_tokens_plan(int fmt, int K, const int* N, int nseg, int gate_up, int M, int sms,
                                            int smem, int* stages, int* groups, int* tiles, int* total) {
  HB_REQUIRE(N && stages && groups && tiles && total && (fmt == HB200_FMT_Q4_K || fmt == HB200_FMT_Q8_0) &&
                 (!gate_up || nseg == 2) && smem > 0,
             "kquant (few-token plan): bad argument");
  for (int s = 0; s < nseg; ++s) HB_REQUIRE(N[s] >= 1, "kquant (few-token plan): tensor %d has no rows", s);
  SbPlan p;
  if (!sb_plan(fmt, K, N, nseg, gate_up, M, sms, smem, &p)) return HB200_ERR_UNSUPPORTED;
  for (int s = 0; s < nseg; ++s) {
    stages[s] = p.stages[s];
    groups[s] = p.groups[s];
    tiles[s] = p.tiles[s];
    total[s] = p.total[s];
  }
  return HB200_OK;
}

template <int FMT, int NTL>
static int sb_launch(hb200_ctx* ctx, const SbParams& p, const SbPlan& plan, cudaStream_t st) {
  static_assert(SbCfg<FMT, NTL>::kB == NTL * 4608 && SbCfg<FMT, NTL>::kPart == kSbWarps * NTL * 512, "sb_plan");
  const int rc = hb_func_smem(ctx, reinterpret_cast<const void*>(kq_sb_kernel<FMT, NTL>), plan.smem);
  if (rc != HB200_OK) return rc;
  HB_CUDA(launch_pdl(kq_sb_kernel<FMT, NTL>, dim3((unsigned)plan.grid), dim3(kSbThreads), plan.smem, st, ctx->pdl, p));
  return HB200_OK;
}

// 2 to 15 tokens; gu: two tensors of equal shape, gate and up, into segs[0].d_y.  HB200_OK when the
// launches were made, 1 when the call is outside what this path covers, < 0 on error.
// Captured calls without memory of their own are outside: the streaming kernel of kquant.cu keeps
// nothing in the context, so captured branches, and a replay beside an eager stream, may share one.
int hb_kq_sb_run(hb200_ctx* ctx, int fmt, const hb200_kquant_seg* segs, int nseg, int K, int gu, const float* d_x,
                 int M, const float* pre_base, const float* pre_gamma, float* pre_out, const float* gamma, float eps,
                 uint8_t* frag, cudaStream_t st) {
  const int NTL = M <= 8 ? 1 : 2, nsb = K / 256;
  int N[kSbMaxSeg] = {};
  for (int s = 0; s < nseg && s < kSbMaxSeg; ++s) N[s] = segs[s].N;
  SbPlan plan;
  if (!sb_plan(fmt, K, N, nseg, gu, M, ctx->sm_count, ctx->smem_optin, &plan)) return 1;
  TcEncodeTiledFn encode = tc_tensor_map_encoder();
  if (encode == nullptr) return 1;
  std::optional<ScratchUse> use;
  if (frag == nullptr) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) {
      cudaGetLastError();
      return 1;
    }
    if (cs != cudaStreamCaptureStatusNone) return 1;
    use.emplace(ctx, st);
    frag = static_cast<uint8_t*>(ctx->d_scratch) + kScratchLmSplit;
  }
  const int unit = fmt == HB200_FMT_Q4_K ? 144 : 272;
  SbParams p = {};
  int cta0 = 0;
  for (int s = 0; s < nseg; ++s) {
    const hb200_kquant_seg& g = segs[s];
    // Q4_K: bytes; Q8_0: 32-bit words (a box dimension holds at most 256 elements, 272 > 256)
    const int esz = fmt == HB200_FMT_Q4_K ? 1 : 4;
    const int rowbytes = nsb * unit;
    const cuuint64_t dims[2] = {(cuuint64_t)(rowbytes / esz), (cuuint64_t)g.N};
    const cuuint64_t strides[1] = {(cuuint64_t)rowbytes};
    const cuuint32_t box[2] = {(cuuint32_t)(unit / esz), (cuuint32_t)plan.rp[s]};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult rc =
        encode(&p.tmap[s], esz == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_UINT32, 2,
               const_cast<void*>(g.d_blocks), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    HB_REQUIRE(rc == CUDA_SUCCESS, "kquant (few tokens): cuTensorMapEncodeTiled failed (%d)", (int)rc);
    p.seg[s] = {g.d_residual,  g.d_y,         g.N,           cta0, plan.ctas[s], plan.rp[s], plan.tiles[s],
                plan.groups[s], plan.stages[s]};
    if (!gu) cta0 += plan.ctas[s];
  }
  p.nseg = nseg;
  p.gu = gu;
  p.nsb = nsb;
  p.M = M;
  p.wbytes = plan.wbytes;
  p.xb = frag;
  p.status = ctx->d_status;
  static_assert(hb_kq_frag_bytes(65536) <= kScratchRowScale - kScratchLmSplit, "fragments in the scratch");
  const int rc = hb_kq_stage_i8(ctx, fmt, K, NTL, d_x, M, pre_base, pre_gamma, pre_out, gamma, eps, frag, st);
  if (rc != HB200_OK) return rc;
  if (fmt == HB200_FMT_Q4_K) return NTL == 1 ? sb_launch<12, 1>(ctx, p, plan, st) : sb_launch<12, 2>(ctx, p, plan, st);
  return NTL == 1 ? sb_launch<8, 1>(ctx, p, plan, st) : sb_launch<8, 2>(ctx, p, plan, st);
}
