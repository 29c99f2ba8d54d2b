// attention_prefill.cu -- causal GQA attention of a prompt chunk on the 5th-generation tensor cores;
// chunks too small for it go to attention_prefill_mma.cu (pf_use_mma).
//
// T new query tokens per sequence against the f16 KV cache that already holds them (the role
// of the reference's batched prefill kernels, flashAttentionBatchKernelF16 and its SWA variant,
// Hesper/WGSL/FlashAttention.lean:601,1621-1624; math of flashAttentionSpec, :60-90).  A CTA owns
// 128 query rows -- 128 / G consecutive tokens times the G query heads of one KV head -- and walks
// the positions those tokens see in tiles of 64, so a K/V tile is read once per 128 / G tokens.
//
//   * warp 4: K and V tiles by 2-D tensor-map TMA (boxes of 64 positions x 64 dims, 128-byte
//     swizzle) into one ring of shared-memory slots, K(j), V(j) alternating.  A tile of a ring
//     cache never spans the wrap: the positions are walked as at most two runs of slots.
//   * warp 5: tcgen05.mma kind::f16.  S(j) = Q K^T with Q in TENSOR MEMORY (pre-multiplied by
//     scale * log2 e, f16) and K as the K-major operand; O += P V with P in tensor memory (it
//     replaces the S it came from) and V, as it lies in the cache, as the MN-major operand.
//     S has two buffers: S(j+1) runs while the softmax works on S(j).
//   * warps 0-3: one thread per row.  Online softmax in the exp2 domain.  The reference maximum of a
//     row moves only when a tile exceeds it by more than 2^8 (P then stays below 2^8, far inside
//     f16): O is rescaled in tensor memory a few times per row instead of once per tile, and the
//     quotient O / l is the same.  P is two f16 terms, what was rounded and what that lost: the
//     maximum of a tile no longer weighs exactly 1, which with one term raised the error against an
//     f64 evaluation by 5 % on average (10 % at most); with two it is 0.77 of what it was, the query's
//     f16 rounding alone, for 14 % more time (256-token chunk at 8192 positions 31 -> 35.6 us).
//   * a row's visible positions are [max(0, pos - window + 1), pos] with pos the token's own
//     position: causal inside the chunk, sliding window if asked.
//
// Tensor memory at D = 256: O 256 columns, Q 128, S 2 x 64 = all 512.  What bounds it: a tile is
// 16 MMAs of N=64 plus 8 of N=256, 1536 cycles of the tensor pipe (the four for P's second term
// show in full), with the softmax's 64 exponentials per row (512 cycles of the special-function
// unit) beside it; K and V come from L2 at 64 KB per tile.  When the query tiles leave SMs
// idle the positions are dealt to several CTAs and a second kernel merges their partials.
#include <math_constants.h>

#include "attention_prefill.cuh"
#include "tcgen05.cuh"

namespace hb {

constexpr int kPfRows = 128;   // query rows per CTA = MMA M
constexpr int kPfTile = 64;    // positions per K/V tile
constexpr int kPfThreads = 192;
constexpr int kPfMaxSplits = 16;

struct PfParams {
  CUtensorMap tmk, tmv;    // caches as [nseq * Hkv * slots][D], boxes of 64 rows x 64 dims
  const void* q;           // [nseq][T][H][D] f32 or f16
  const int32_t* seqlens;  // [nseq] lengths after the T tokens
  float* out;              // [nseq][T][H][D]
  int q_is_f16;
  int nseq, T, H, Hkv, G, slots, window, ring;
  int out_bulk;            // out is 16-byte aligned: rows leave by bulk copies, else by float2 stores
  float scale_log2;
  // nsplit > 1: the K/V tiles of a query tile are dealt to nsplit CTAs; each writes its
  // unnormalised partial and its (max, sum), attn_prefill_merge_kernel combines them
  int nsplit;
  float* part_o;   // [nseq][T][H][nsplit][D]
  float* part_ml;  // [nseq][T][H][nsplit][2]  (max in the exp2 domain, sum)
  uint32_t* status;
};

template <int D>
struct PfCfg {
  static constexpr int kO0 = 0, kQ0 = D, kS0 = D + D / 2;   // tensor-memory columns
  static constexpr int kCols = D == 256 ? 512 : (D == 128 ? 512 : 256);
  static constexpr int kSlotBytes = kPfTile * D * 2;        // one K or V tile: 32 / 16 / 8 KB
  static constexpr int kBoxBytes = kPfTile * 128;
  static constexpr int kSlots = 6;
  static constexpr int kOutStride = D * 4 + 16;             // padded f32 row of the epilogue
  static constexpr int kRing = kSlots * kSlotBytes;
  static constexpr int kData = kRing > kPfRows * kOutStride ? kRing : kPfRows * kOutStride;
  // D = 128 takes all of tensor memory: a second CTA of an SM, placed there early beside the kernel
  // before, would only wait for the first.  More than half of the shared memory keeps it off.
  static constexpr int kSmem = D == 128 ? 118784 : 1024 + kData;
  static_assert(1024 + kData <= kSmem, "shared memory of a CTA");
  static constexpr uint32_t kIdescS = (1u << 4) | ((uint32_t)(kPfTile >> 3) << 17) | ((uint32_t)(kPfRows >> 4) << 24);
  // B (= V) is MN-major
  static constexpr uint32_t kIdescO =
      (1u << 4) | (1u << 16) | ((uint32_t)(D >> 3) << 17) | ((uint32_t)(kPfRows >> 4) << 24);
  static_assert(kS0 + 2 * kPfTile <= kCols, "tensor memory columns");
  static_assert(kSmem <= 232448, "shared memory");
};

// One tile of the walk: first position, its slot, and how many of the 64 are real.
struct PfTileAt {
  int pos, slot, n;
};
// The positions [lo, hi] as at most two runs of slots (a ring wraps once at most, window + T - 1
// <= slots), each cut into tiles from its own start.
struct PfWalk {
  int lo, hi, slot0, run0, tiles0, tiles;
  __device__ __forceinline__ PfWalk(int lo_, int hi_, int slots, int ring) : lo(lo_), hi(hi_) {
    const int n = hi >= lo ? hi - lo + 1 : 0;
    slot0 = ring ? lo % slots : lo;
    run0 = ring ? min(n, slots - slot0) : n;
    tiles0 = (run0 + kPfTile - 1) / kPfTile;
    tiles = tiles0 + (n - run0 + kPfTile - 1) / kPfTile;
  }
  __device__ __forceinline__ PfTileAt at(int j) const {
    if (j < tiles0) return {lo + j * kPfTile, slot0 + j * kPfTile, min(kPfTile, run0 - j * kPfTile)};
    const int k = j - tiles0, p = lo + run0 + k * kPfTile;
    return {p, k * kPfTile, min(kPfTile, hi - p + 1)};
  }
};

__device__ __forceinline__ float pf_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pf_pack(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

template <int D>
__global__ void __launch_bounds__(kPfThreads, 1)
    attn_prefill_tiled_kernel(const __grid_constant__ PfParams p) {
  using Cfg = PfCfg<D>;
  constexpr int kSlots = Cfg::kSlots;
  constexpr int kCopyWarp = 4, kMmaWarp = 5;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  uint64_t* kv_full = reinterpret_cast<uint64_t*>(smem);  // [kSlots] tile landed
  uint64_t* kv_free = kv_full + kSlots;  // [kSlots] the MMAs that read it have retired
  uint64_t* s_full = kv_free + kSlots;   // [2] S(j) complete
  uint64_t* p_full = s_full + 2;         // [2] P(j) written by the four softmax warps
  uint64_t* q_full = p_full + 2;         // [1] Q in tensor memory
  uint64_t* o_done = q_full + 1;         // [2] P V(j) has retired, even and odd j: a parity tells a
                                         // product from the one two before it, not from the next
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 2);
  uint8_t* ring = smem + 1024;

  const int G = p.G, TQ = kPfRows / G;
  const int qt = blockIdx.x / p.nsplit, split = blockIdx.x % p.nsplit;
  const int kvh = blockIdx.y, b = blockIdx.z;

  if (tid == 0) {
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_free[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 4);
      mbar_init(&o_done[i], 1);
    }
    mbar_init(q_full, 4);
    fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)), "n"(Cfg::kCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_before_sync();
  __syncthreads();
  tc_after_sync();
  const uint32_t tmem = *tmem_slot;
  pdl_trigger();
  pdl_wait();  // q, the cache rows of this chunk and seqlens come from earlier kernels

  int len = max(p.seqlens[b], 0);  // positions after the chunk
  if (!p.ring) len = min(len, p.slots);  // a corrupt length never overruns a linear cache
  const int t0 = qt * TQ;                // first token of this CTA
  const int t1 = min(t0 + TQ, p.T) - 1;  // last one
  // positions of the chunk's tokens: token t sits at len - T + t
  const int pos_first = len - p.T + t0, pos_last = len - p.T + t1;
  const int kv_lo = p.window > 0 ? max(0, pos_first - p.window + 1) : 0;
  const PfWalk walk(kv_lo, pos_last, p.slots, p.ring);
  // this CTA's share of the tiles
  const int tps = (walk.tiles + p.nsplit - 1) / p.nsplit;
  const int j0 = split * tps;
  const int ntiles = max(0, min(walk.tiles, j0 + tps) - j0);
  bool ok = true;

  if (warp == kCopyWarp) {
    // ================= K and V tiles ============================================================
    const int row0 = (b * p.Hkv + kvh) * p.slots;
    TcRing<kSlots> r;
    for (int i = 0; i < 2 * ntiles && ok; ++i, r.advance()) {
      ok = tc_wait_w(&kv_free[r.i], r.phase ^ 1, p.status);
      if (!ok) break;
      if (tc_elect()) {
        const CUtensorMap* tm = i & 1 ? &p.tmv : &p.tmk;
        const PfTileAt t = walk.at(j0 + (i >> 1));
        uint8_t* dst = ring + (size_t)r.i * Cfg::kSlotBytes;
        mbar_arrive_expect_tx(&kv_full[r.i], Cfg::kSlotBytes);
#pragma unroll
        for (int c = 0; c < D / 64; ++c)
          asm volatile(
              "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
              " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst + c * Cfg::kBoxBytes)),
              "l"(reinterpret_cast<uint64_t>(tm)), "r"(c * 64), "r"(row0 + t.slot), "r"(smem_u32(&kv_full[r.i]))
              : "memory");
      }
      __syncwarp();
    }
  } else if (warp == kMmaWarp) {
    // ================= MMA issue: the whole warp runs the loop, one lane issues =================
    TcRing<kSlots> r;  // slot of K(j + 1), then of V(j)
    const uint32_t kdesc0 = tc_desc_lo(smem_u32(ring), 16), vdesc0 = tc_desc_lo(smem_u32(ring), Cfg::kBoxBytes);
    constexpr uint32_t kSw = 2u << 29;  // 128-byte swizzle
    auto scores = [&](int j) {
      ok = ok && tc_wait_w(&kv_full[r.i], r.phase, p.status);
      if (!ok) return;
      tc_after_sync();
      const uint32_t kd = kdesc0 + r.i * (Cfg::kSlotBytes >> 4);
#pragma unroll
      for (int m = 0; m < D / 16; ++m)
        tc_mma_f16_ta_w<tc_desc_hi(1024) | kSw, Cfg::kIdescS>(
            tmem + Cfg::kS0 + (j & 1) * kPfTile, tmem + Cfg::kQ0 + m * 8,
            kd + (((m >> 2) * Cfg::kBoxBytes + (m & 3) * 32) >> 4), m > 0 ? 1u : 0u);
      tc_commit_w(&s_full[j & 1]);
      tc_commit_w(&kv_free[r.i]);
    };
    ok = tc_wait_w(q_full, 0, p.status);
    // slots go K(0), V(0), K(1), V(1), ...: the score product of tile j + 1 skips over V(j)
    if (ntiles > 0) scores(0);
    uint32_t vi = 1, vphase = 0;  // slot of V(j)
    for (int j = 0; j < ntiles && ok; ++j) {
      if (j + 1 < ntiles) {
        r.advance(2);
        scores(j + 1);
      }
      ok = ok && tc_wait_w(&p_full[j & 1], (uint32_t)((j >> 1) & 1), p.status);
      ok = ok && tc_wait_w(&kv_full[vi], vphase, p.status);
      if (!ok) break;
      tc_after_sync();
      const uint32_t vd = vdesc0 + vi * (Cfg::kSlotBytes >> 4);
#pragma unroll
      for (int m = 0; m < kPfTile / 8; ++m)  // the weights' f16 terms, then what they lost
        tc_mma_f16_ta_w<tc_desc_hi(1024) | kSw, Cfg::kIdescO>(
            tmem + Cfg::kO0, tmem + Cfg::kS0 + (j & 1) * kPfTile + m * 8,
            vd + (((m % (kPfTile / 16)) * 2048) >> 4), (j > 0 || m > 0) ? 1u : 0u);
      tc_commit_w(&kv_free[vi]);
      tc_commit_w(&o_done[j & 1]);
      vi += 2;
      if (vi >= kSlots) {
        vi -= kSlots;
        vphase ^= 1;
      }
    }
  } else {
    // ================= softmax: one thread per row ================================================
    const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
    const int row = tid;  // 0..127
    const int t = t0 + row / G, h = kvh * G + row % G;
    const bool live = t < p.T;
    const int pos = len - p.T + t;
    const int lo = p.window > 0 ? max(0, pos - p.window + 1) : 0;
    // ---- Q row, scaled, f16, into tensor memory (rows past T are zero) ---------------------------
    {
      const size_t qi = (((size_t)b * p.T + (live ? t : 0)) * p.H + h) * D;
#pragma unroll 1
      for (int c = 0; c < D; c += 64) {
        uint32_t w[32];
        if (p.q_is_f16) {
          const __half2* q2 = reinterpret_cast<const __half2*>(static_cast<const __half*>(p.q) + qi + c);
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const float2 v = __half22float2(q2[i]);
            w[i] = live ? pf_pack(v.x * p.scale_log2, v.y * p.scale_log2) : 0u;
          }
        } else {
          const float4* q4 = reinterpret_cast<const float4*>(static_cast<const float*>(p.q) + qi + c);
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float4 v = q4[i];
            w[2 * i] = live ? pf_pack(v.x * p.scale_log2, v.y * p.scale_log2) : 0u;
            w[2 * i + 1] = live ? pf_pack(v.z * p.scale_log2, v.w * p.scale_log2) : 0u;
          }
        }
        HB_TMEM_ST32(lane_base + (uint32_t)(Cfg::kQ0 + c / 2), w);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(q_full);
    }

    // P V(i) has retired; asked behind s_full(i + 1) or, of the last product, s_full(i).  S(j) was issued
    // behind P V(j - 2), so the barrier's phase is i's own or the one after it: a parity tells these
    // apart.  With one barrier for all products a warp that came late to the end of the walk
    // asked for the phase before last and waited in vain.
    auto product_done = [&](int i) {
      ok = ok && tc_wait_w(&o_done[i & 1], (uint32_t)((i >> 1) & 1), p.status);
    };
    float m = -CUDART_INF_F, l = 0.f;  // reference maximum and sum of the row
    for (int j = 0; j < ntiles; ++j) {
      const PfTileAt at = walk.at(j0 + j);
      if (at.n < kPfTile) {
        // Rows of V past the run's end are whatever the cache holds there, NaN included, and P = 0
        // does not silence that: zero them before P(j) releases the product (at most two tiles of
        // a walk).
        const int slot = (2 * j + 1) % kSlots;
        ok = ok && tc_wait_w(&kv_full[slot], (uint32_t)(((2 * j + 1) / kSlots) & 1), p.status);
        for (int i = tid; i < (kPfTile - at.n) * (D / 8); i += 128) {
          const int rr = at.n + i / (D / 8), u = i % (D / 8);
          *reinterpret_cast<uint4*>(ring + (size_t)slot * Cfg::kSlotBytes + (u >> 3) * Cfg::kBoxBytes + rr * 128 +
                                    ((u & 7) << 4)) = make_uint4(0, 0, 0, 0);
        }
        fence_proxy_async();
      }
      ok = ok && tc_wait_w(&s_full[j & 1], (uint32_t)((j >> 1) & 1), p.status);
      tc_after_sync();
      const uint32_t s_addr = lane_base + (uint32_t)(Cfg::kS0 + (j & 1) * kPfTile);
      uint32_t v0[32], v1[32];
      HB_TMEM_LD32(v0, s_addr);
      HB_TMEM_LD32(v1, s_addr + 32);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      // positions of this tile that the row sees: [a, e)
      const int a = max(lo - at.pos, 0), e = live ? min(pos - at.pos + 1, at.n) : 0;
      if (a > 0 || e < kPfTile) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          if (i < a || i >= e) v0[i] = 0xff800000u;  // -inf
          if (i + 32 < a || i + 32 >= e) v1[i] = 0xff800000u;
        }
      }
      float mx[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
      for (int i = 0; i < 32; ++i) mx[i & 3] = fmaxf(mx[i & 3], fmaxf(__uint_as_float(v0[i]), __uint_as_float(v1[i])));
      const float mt = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      const bool grow = mt > m + 8.f;  // also the first visible tile: m = -inf
      if (j > 0 && __any_sync(0xffffffffu, grow)) {
        // rescale O once P V(j - 1) has retired
        product_done(j - 1);
        tc_after_sync();
        const float alpha = grow ? pf_exp2(m - mt) : 1.f;  // m = -inf: 0
#pragma unroll 1
        for (int c = 0; c < D; c += 32) {
          uint32_t o[32];
          HB_TMEM_LD32(o, lane_base + (uint32_t)(Cfg::kO0 + c));
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          HB_TMEM_ST32(lane_base + (uint32_t)(Cfg::kO0 + c), o);
        }
        l *= alpha;
      }
      if (grow) m = mt;
      const float base = m == -CUDART_INF_F ? 0.f : m;  // nothing visible yet: avoid inf - inf
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t pk[32], lo16[32];
      auto two_terms = [&](int i, float x, float y) {
        pk[i] = pf_pack(x, y);
        const float2 r = __half22float2(*reinterpret_cast<const __half2*>(&pk[i]));
        lo16[i] = pf_pack(x - r.x, y - r.y);
      };
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float e0 = pf_exp2(__uint_as_float(v0[2 * i]) - base), e1 = pf_exp2(__uint_as_float(v0[2 * i + 1]) - base);
        const float e2 = pf_exp2(__uint_as_float(v1[2 * i]) - base), e3 = pf_exp2(__uint_as_float(v1[2 * i + 1]) - base);
        sum[0] += e0;
        sum[1] += e1;
        sum[2] += e2;
        sum[3] += e3;
        two_terms(i, e0, e1);
        two_terms(16 + i, e2, e3);
      }
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      HB_TMEM_ST32(s_addr, pk);
      HB_TMEM_ST32(s_addr + 32, lo16);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[j & 1]);
    }

    // ---- O out of tensor memory, normalised or as a partial; whole rows by bulk copies -----------
    if (ntiles > 0) product_done(ntiles - 1);  // products retire in order
    tc_after_sync();
    const float f = p.nsplit > 1 ? 1.f : (l > 0.f ? 1.f / l : 0.f);
    // the K/V ring is idle now: every product has retired
    float* orow = reinterpret_cast<float*>(ring + (size_t)row * Cfg::kOutStride);
#pragma unroll 1
    for (int c = 0; c < D; c += 32) {
      uint32_t o[32];
      if (ntiles > 0) {
        HB_TMEM_LD32(o, lane_base + (uint32_t)(Cfg::kO0 + c));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = 0u;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
        *reinterpret_cast<float4*>(orow + c + 4 * i) =
            make_float4(__uint_as_float(o[4 * i]) * f, __uint_as_float(o[4 * i + 1]) * f,
                        __uint_as_float(o[4 * i + 2]) * f, __uint_as_float(o[4 * i + 3]) * f);
    }
    fence_proxy_async();
    if (live) {
      const size_t ri = ((size_t)b * p.T + t) * p.H + h;
      float* dst = p.nsplit > 1 ? p.part_o + (ri * p.nsplit + split) * D : p.out + ri * D;
      if (p.nsplit > 1 || p.out_bulk) {
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(orow)),
                     "n"(D * 4)
                     : "memory");
      } else {
        for (int c = 0; c < D; c += 2)
          *reinterpret_cast<float2*>(dst + c) = *reinterpret_cast<const float2*>(orow + c);
      }
      if (p.nsplit > 1)
        *reinterpret_cast<float2*>(p.part_ml + (ri * p.nsplit + split) * 2) = make_float2(m, l);
    }
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  tc_before_sync();
  __syncthreads();
  if (warp == kMmaWarp)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(Cfg::kCols));
}

// out = sum_s 2^(m_s - m*) O_s / sum_s 2^(m_s - m*) l_s over the splits of one (token, head): a
// warp per row, lane s holding split s's weight.
template <int D>
__global__ void __launch_bounds__(256) attn_prefill_merge_kernel(const float* part_o, const float* part_ml,
                                                                 int nsplit, long rows, float* out) {
  pdl_trigger();
  pdl_wait();
  constexpr int V = D / 32;  // floats per lane
  const int lane = threadIdx.x & 31;
  const long row = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= rows) return;
  float2 ml = make_float2(-CUDART_INF_F, 0.f);
  if (lane < nsplit) ml = __ldcg(reinterpret_cast<const float2*>(part_ml + row * nsplit * 2) + lane);
  const float mstar = warp_max(ml.x);
  const float w = ml.x == -CUDART_INF_F ? 0.f : exp2f(ml.x - mstar);
  const float lsum = warp_sum(w * ml.y);
  const float inv = lsum > 0.f ? 1.f / lsum : 0.f;
  float acc[V];
#pragma unroll
  for (int i = 0; i < V; ++i) acc[i] = 0.f;
#pragma unroll 4
  for (int s = 0; s < nsplit; ++s) {
    const float ws = __shfl_sync(0xffffffffu, w, s);
    const float2* src = reinterpret_cast<const float2*>(part_o + (row * nsplit + s) * D) + lane;
#pragma unroll
    for (int i = 0; i < V / 2; ++i) {
      const float2 x = __ldcg(src + 32 * i);
      acc[2 * i] += ws * x.x;
      acc[2 * i + 1] += ws * x.y;
    }
  }
  float2* dst = reinterpret_cast<float2*>(out + row * D) + lane;
#pragma unroll
  for (int i = 0; i < V / 2; ++i) dst[32 * i] = make_float2(acc[2 * i] * inv, acc[2 * i + 1] * inv);
}

}  // namespace hb

using namespace hb;

// How many CTAs share the K/V range of a query tile: as many as there are SMs for in one wave,
// but no split shorter than 4 tiles of the longest range a tile can see.  A function of the
// shapes only (the workspace is sized with it).
static int pf_pick_splits(const hb200_ctx* ctx, int nseq, int T, int H, int Hkv, int slots, int window) {
  const int G = H / Hkv, TQ = kPfRows / G;
  const long ctas = (long)((T + TQ - 1) / TQ) * Hkv * nseq;
  long span = slots;
  if (window > 0 && (long)window + T < span) span = (long)window + T;
  long ns = ctx->sm_count / ctas;
  const long most = (span + kPfTile - 1) / kPfTile / 4;
  if (ns > most) ns = most;
  if (ns > kPfMaxSplits) ns = kPfMaxSplits;
  return ns < 1 ? 1 : (int)ns;
}

// Positions of a cache that the tokens of a chunk see between them, at most.
static long pf_span(int T, int slots, int window) {
  return window > 0 && (long)window + T < slots ? (long)window + T : slots;
}

// Whether the mma.sync kernel (attention_prefill_mma.cu) takes a chunk.  The kernel here costs more to
// start, holds an SM by itself and, at 128 rows a CTA, has half as many of them to deal; its tiles
// are the cheaper the wider the head.  Device times over 223 shapes (1 to 20 KV heads x sequences of 4
// query heads, 8 to 400 tokens, 16 to 8000 positions) give, in us,
//   here  5.8 + 1.15 t w    D = 128: 7.8 + 1.2 t w     t tiles of a CTA, w waves of CTAs
//   mma   3.8 + (0.47 + 0.72 c) t    5.8 + (0.62 + 1.05 c) t    c CTAs per SM, at least 1
// and for the merge of splits 1.8 + 0.8 and 1.4 + 2.6 (1.5 + 1.0 and 0.8 + 1.75) per MB of partials,
// within 10 %.  Measured, mma / here: D = 64 8 tokens x 16 positions 4.8 / 6.7, 40 x 300 9.3 / 11.0,
// 20 pairs 100 x 8000 109 / 154, but 400 x 8000 40.5 / 22.1; D = 128 40 x 80 9.6 / 12.1, 400 x 1000 17.3 /
// 16.0.  D = 256: only where a tile or two are all there is, 40 x 80 14.8 / 18.3, 16 x 300 21.7 / 16.5.
static bool pf_use_mma(const hb200_ctx* ctx, int nseq, int T, int H, int Hkv, int D, int slots, int window) {
  const long span = pf_span(T, slots, window);
  if (D == 256) return span <= 128;
  const int G = H / Hkv, sms = ctx->sm_count;
  const float mb = (float)nseq * T * H * D * 4e-6f;
  auto qtiles = [&](int rows) { return (long)((T + rows / G - 1) / (rows / G)) * Hkv * nseq; };
  const long tiles = (span + 63) / 64, cn = qtiles(kPfRows), co = qtiles(kPmRows);
  const int nn = pf_pick_splits(ctx, nseq, T, H, Hkv, slots, window);
  const int no = hb_attn_prefill_mma_splits(ctx, nseq, T, G, Hkv, D, span);
  const float tn = (float)((tiles + nn - 1) / nn * ((cn * nn + sms - 1) / sms));
  const float to = (float)((tiles + no - 1) / no), c = fmaxf(1.f, (float)(co * no) / sms);
  const bool d64 = D == 64;
  const float here = (d64 ? 5.8f + 1.15f * tn : 7.8f + 1.2f * tn) +
                     (nn > 1 ? (d64 ? 1.8f + 0.8f * nn * mb : 1.5f + 1.0f * nn * mb) : 0.f);
  const float mma = (d64 ? 3.8f + (0.47f + 0.72f * c) * to : 5.8f + (0.62f + 1.05f * c) * to) +
                    (no > 1 ? (d64 ? 1.4f + 2.6f * no * mb : 0.8f + 1.75f * no * mb) : 0.f);
  return mma < here;
}

size_t hb_attn_prefill_tiled_ws(const hb200_ctx* ctx, int nseq, int T, int H, int Hkv, int D,
                                int slots) {
  if (H % Hkv || H / Hkv > 8) return 0;
  // of the kernels' split counts the larger one: a window may change which of them runs
  int ns = pf_pick_splits(ctx, nseq, T, H, Hkv, slots, 0);
  const int no = hb_attn_prefill_mma_splits(ctx, nseq, T, H / Hkv, Hkv, D, slots);
  if (no > ns) ns = no;
  return ns > 1 ? (size_t)nseq * T * H * ns * ((size_t)D + 2) * sizeof(float) + 256 : 0;
}

template <int D>
static int pf_launch(hb200_ctx* ctx, const PfParams& p, dim3 grid, cudaStream_t st) {
  const int rc = hb_func_smem(ctx, reinterpret_cast<const void*>(attn_prefill_tiled_kernel<D>), PfCfg<D>::kSmem);
  if (rc) return rc;
  HB_CUDA(launch_pdl(attn_prefill_tiled_kernel<D>, grid, dim3(kPfThreads), (size_t)PfCfg<D>::kSmem, st,
                     ctx->pdl, p));
  return HB200_OK;
}

static int pf_merge(hb200_ctx* ctx, const float* part_o, const float* part_ml, int nsplit, long rows, int D,
                    float* out, cudaStream_t st) {
  auto kern = D == 64 ? attn_prefill_merge_kernel<64> : (D == 128 ? attn_prefill_merge_kernel<128>
                                                                  : attn_prefill_merge_kernel<256>);
  HB_CUDA(launch_pdl(kern, dim3((unsigned)((rows + 7) / 8)), dim3(256), 0, st, ctx->pdl, part_o, part_ml, nsplit,
                     rows, out));
  return HB200_OK;
}

// Causal attention of T query tokens per sequence on a tiled kernel.  HB200_OK when the
// launch was made, 1 when the shape is outside what it covers (the caller runs every token as a
// decode query instead), < 0 on error.
int hb_attn_prefill_tiled(hb200_ctx* ctx, const void* d_q, int q_is_f16, const void* d_k,
                          const void* d_v, const int32_t* d_seqlens, int nseq, int T, int H,
                          int Hkv, int D, int slots, int window, int ring, float scale,
                          void* d_ws, size_t ws_bytes, float* d_out, cudaStream_t st) {
  const int G = H / Hkv;
  if (!(G == 1 || G == 2 || G == 4 || G == 8)) return 1;
  if (!(D == 64 || D == 128 || D == 256)) return 1;
  if (nseq > 65535 || Hkv > 65535) return 1;
  if (q_is_f16 ? (reinterpret_cast<uintptr_t>(d_q) & 3) : (reinterpret_cast<uintptr_t>(d_q) & 15)) return 1;
  if (reinterpret_cast<uintptr_t>(d_out) & 7) return 1;
  TcEncodeTiledFn encode = tc_tensor_map_encoder();
  const bool mma = encode == nullptr || (long)nseq * Hkv * slots >= (1l << 31) ||  // rows of a tensor map
                   pf_use_mma(ctx, nseq, T, H, Hkv, D, slots, window);
  int nsplit = mma ? hb_attn_prefill_mma_splits(ctx, nseq, T, G, Hkv, D, pf_span(T, slots, window))
                   : pf_pick_splits(ctx, nseq, T, H, Hkv, slots, window);
  if (nsplit > 1) {
    // never more than the workspace holds (a caller may have sized it for another T)
    const size_t per = (size_t)nseq * T * H * ((size_t)D + 2) * sizeof(float);
    if (d_ws == nullptr || (reinterpret_cast<uintptr_t>(d_ws) & 15)) nsplit = 1;
    else if ((size_t)nsplit * per > ws_bytes) nsplit = ws_bytes / per < 1 ? 1 : (int)(ws_bytes / per);
  }
  const long rows = (long)nseq * T * H;
  float* const part_o = nsplit > 1 ? static_cast<float*>(d_ws) : nullptr;
  float* const part_ml = nsplit > 1 ? part_o + (size_t)rows * nsplit * D : nullptr;
  const float scale_log2 = scale * 1.4426950408889634f;
  int rc;
  if (mma) {
    const PmParams p = {d_q, static_cast<const __half*>(d_k), static_cast<const __half*>(d_v), d_seqlens, d_out,
                        q_is_f16, nseq, T, H, Hkv, G, slots, window, ring, scale_log2, nsplit, part_o, part_ml};
    rc = hb_attn_prefill_mma(ctx, p, D, st);
    return rc || nsplit == 1 ? rc : pf_merge(ctx, part_o, part_ml, nsplit, rows, D, d_out, st);
  }
  PfParams p = {};
  const cuuint64_t dims[2] = {(cuuint64_t)D, (cuuint64_t)nseq * Hkv * slots};
  const cuuint64_t strides[1] = {(cuuint64_t)D * 2};
  const cuuint32_t box[2] = {64, kPfTile};
  const cuuint32_t estr[2] = {1, 1};
  for (int i = 0; i < 2; ++i) {
    const CUresult erc = encode(i ? &p.tmv : &p.tmk, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                                const_cast<void*>(i ? d_v : d_k), dims, strides, box, estr,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    HB_REQUIRE(erc == CUDA_SUCCESS, "attn (prefill): cuTensorMapEncodeTiled failed (%d)", (int)erc);
  }
  p.q = d_q;
  p.seqlens = d_seqlens;
  p.out = d_out;
  p.q_is_f16 = q_is_f16;
  p.nseq = nseq;
  p.T = T;
  p.H = H;
  p.Hkv = Hkv;
  p.G = G;
  p.slots = slots;
  p.window = window;
  p.ring = ring;
  p.out_bulk = (reinterpret_cast<uintptr_t>(d_out) & 15) == 0;
  p.scale_log2 = scale_log2;
  p.status = ctx->d_status;
  p.nsplit = nsplit;
  p.part_o = part_o;
  p.part_ml = part_ml;
  const int TQ = kPfRows / G;
  const dim3 grid((unsigned)((T + TQ - 1) / TQ) * p.nsplit, (unsigned)Hkv, (unsigned)nseq);
  rc = D == 64 ? pf_launch<64>(ctx, p, grid, st)
       : D == 128 ? pf_launch<128>(ctx, p, grid, st)
                  : pf_launch<256>(ctx, p, grid, st);
  return rc || nsplit == 1 ? rc : pf_merge(ctx, part_o, part_ml, nsplit, rows, D, d_out, st);
}
