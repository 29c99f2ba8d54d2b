// lmhead_mma.cu -- batched (16..64 tokens) LM head on the 5th-generation tensor cores.
//
// logits[m][v] = sum_k table[v][k] * xn[m][k] with the 16-bit table (bf16 or f16, [V][K], the
// tied embedding of Hesper/Models/BitNet.lean:456) and f32 activations, optional final RMSNorm
// in front and the greedy argmax (first strict maximum, Hesper/Inference/Sampling.lean:74)
// behind.  The batch-1 kernel streams the table once per 8 tokens and is FMA-bound from 16
// tokens on; here the table is streamed ONCE and the contraction runs as tcgen05.mma
// kind::f16 with f32 accumulators in tensor memory.
//
// Keeping f32-activation accuracy on a 16-bit tensor-core path: each activation is split as
// x = hi + lo with hi = round16(x), lo = round16(x - hi).  Products of 16-bit values are exact
// in the f32 accumulator, so the logit error is that of dropping x - hi - lo (2^-17 relative
// for bf16, 2^-22 for f16) plus the accumulation order.  With TS = 32 or 64 token slots hi and lo
// are the token rows 0..TS-1 and TS..2TS-1 of one N = 2 TS operand; the epilogue adds the halves.
//
//   lm_split_kernel     one CTA per token slot: optional RMSNorm, split, and store in the
//                       shared-memory operand layout (K-major 8x16-byte core matrices), one
//                       block per 64-wide K block
//   lmhead_mma_kernel   one CTA per SM with a contiguous share of the 128-row tiles, in rounds of
//     512 / N tiles whose accumulators fill tensor memory:
//     warp 0      table boxes [128 rows x 64 el] by 2-D tensor-map TMA (128-byte swizzle), two
//                 per tile and K step (256 bytes of a row together), the tiles of a round side by
//                 side, a ring of its own;
//     warp 1      the K step's activations, ONCE per round: one CTA per tile re-read them for every
//                 tile, as many bytes from L2 as the table itself and half of the ring;
//     warp 2      MMA issue (M=128, K=16): whole warp converged, one lane issues;
//     warps 4-19  epilogue: warp w reads lane quarter w & 3 of the accumulators (w >> 2) - 1, + 4, ...:
//                 hi + lo, optional logits store, argmax over the tile's rows (redux + ballot); one
//                 atomicMax of the ordered (value,row) key per token and CTA.
// HBM-bound.  Measured, V=128256 K=2560, whole call (split, product, argmax): 32 tokens 143 to 149 ->
// 113 to 117 us (5.6 to 5.8 TB/s of table bytes, by the box), of which the product is 106; 64 tokens
// 149 -> 117 in the product; with one box per step 124 and 131 there (half a DRAM burst per row).
// Every mbarrier wait is bounded; on expiry the kernel still releases its tensor memory.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "tcgen05.cuh"

namespace hb {

constexpr int kLmRows = 128;      // vocabulary rows per tile = MMA M
constexpr int kLmBlock = 64;      // elements of a swizzled box = 128 bytes of a table row
constexpr int kLmABox = kLmRows * kLmBlock * 2;  // 16 KB
constexpr int kLmABytes = 2 * kLmABox;           // a pipeline step: 256 bytes of every row
constexpr int kLmEpiWarps = 16;
constexpr int kLmThreads = (4 + kLmEpiWarps) * 32;

template <int TS>
struct LmCfg {
  static constexpr int kN = 2 * TS;
  static constexpr int kTiles = 512 / kN;         // accumulators in tensor memory: tiles of a round
  static constexpr int kBBlock = kN * kLmBlock * 2;
  static constexpr int kBBytes = 2 * kBBlock;
  static constexpr int kAStages = TS == 32 ? 5 : 4;
  static constexpr int kBStages = 2;
  static constexpr int kCtrl = 1024 + TS * kLmEpiWarps * 8;  // barriers, tensor-memory slot; argmax keys
  static constexpr int kSmem = kCtrl + kAStages * kLmABytes + kBStages * kBBytes;
  static_assert(kSmem <= 232448, "shared memory budget of one CTA");
};

struct LmSplitParams {
  const float* x;      // [M][K]
  const float* gamma;  // nullable
  float eps;
  int K, M, dtype;     // dtype 0 = bf16, 1 = f16
  int slots;           // token slots: hi in rows 0..slots-1, lo in slots..2 slots-1 of each block
  uint8_t* xb;         // [K/64] operand blocks
  // f16 table only: the row is divided by a power of two s that brings its largest magnitude
  // into [2^13, 2^14) -- f16 has 5 exponent bits, an activation above 65504 would round to
  // infinity and one below 6e-5 lose bits -- and s is stored here for the product's epilogue
  float* rowscale;     // nullable [M]
};

struct LmMmaParams {
  CUtensorMap tmap;    // table as [V rows][K elements of 2 bytes], boxes of 128 rows x 64
  const uint8_t* xb;
  float* logits;       // nullable [M][V]
  unsigned long long* keys;  // nullable [M]
  long V;
  int K, M, ntiles;
  const float* rowscale;  // nullable [M]: factor the staging divided each token's row by
  uint32_t idesc;
  uint32_t* status;
};

__device__ __forceinline__ uint16_t round16(float v, int dtype) {
  return dtype == 0 ? __bfloat16_as_ushort(__float2bfloat16_rn(v))
                    : __half_as_ushort(__float2half_rn(v));
}
__device__ __forceinline__ float widen16(uint16_t h, int dtype) {
  return dtype == 0 ? __uint_as_float((uint32_t)h << 16) : __half2float(__ushort_as_half(h));
}

__global__ void __launch_bounds__(256) lm_split_kernel(const __grid_constant__ LmSplitParams p) {
  __shared__ double red[8];
  __shared__ float redf[8];
  pdl_trigger();
  // norm weights are constants of the model: into L1 before the wait on the previous kernel
  if (p.gamma)
    for (int i = threadIdx.x * 32; i < p.K; i += 256 * 32)
      asm volatile("prefetch.global.L1 [%0];" ::"l"(p.gamma + i));
  pdl_wait();
  const int m = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int K = p.K;
  // 8 consecutive k of operand row `row` -> their 16 bytes
  auto dst = [&](int row, int k) {
    return p.xb + (size_t)(k >> 6) * p.slots * 256 + (size_t)(row >> 3) * 1024 +
           (size_t)((k & 63) >> 3) * 128 + (size_t)(row & 7) * 16;
  };
  if (m >= p.M) {
    for (int k = tid * 8; k < K; k += 256 * 8) {
      *reinterpret_cast<uint4*>(dst(m, k)) = make_uint4(0, 0, 0, 0);
      *reinterpret_cast<uint4*>(dst(p.slots + m, k)) = make_uint4(0, 0, 0, 0);
    }
    return;
  }
  const float* xg = p.x + (size_t)m * K;
  float inv_s = 1.f;  // 1 / row scale, set before the first emit
  // block-wide: the power of two that brings `amax` into [2^13, 2^14); stores it, returns 1/s
  auto row_scale = [&](float amax) {
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 16));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 8));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    if (lane == 0) redf[warp] = amax;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, redf[i]);
    int e = 13;  // an all-zero (or non-finite) row keeps s = 1
    if (amax > 0.f && amax <= 3.0e38f) e = min(max(ilogbf(amax), -100), 120);
    if (tid == 0) p.rowscale[m] = ldexpf(1.f, e - 13);
    return ldexpf(1.f, 13 - e);
  };
  auto emit = [&](int k, const float (&vin)[8]) {
    uint32_t hi[4], lo[4];
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = vin[e] * inv_s;  // exact: a power of two
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint16_t h[2], l[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        h[e] = round16(v[2 * j + e], p.dtype);
        l[e] = round16(__fsub_rn(v[2 * j + e], widen16(h[e], p.dtype)), p.dtype);
      }
      hi[j] = (uint32_t)h[0] | ((uint32_t)h[1] << 16);
      lo[j] = (uint32_t)l[0] | ((uint32_t)l[1] << 16);
    }
    *reinterpret_cast<uint4*>(dst(m, k)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(dst(p.slots + m, k)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  };
  constexpr int kHeld = 5;  // 8-element groups a thread keeps in registers: K <= 10240
  const bool aligned =
      ((reinterpret_cast<uintptr_t>(xg) | reinterpret_cast<uintptr_t>(p.gamma)) & 15) == 0;
  if (K <= kHeld * 2048 && aligned) {
    // the row is read once and stays in registers between the sum of squares and the rounding
    float v[kHeld][8];
#pragma unroll
    for (int i = 0; i < kHeld; ++i) {
      const int k = tid * 8 + i * 2048;
      const bool in = k < K;
      const float4 a = in ? *reinterpret_cast<const float4*>(xg + k) : make_float4(0, 0, 0, 0);
      const float4 b = in ? *reinterpret_cast<const float4*>(xg + k + 4) : make_float4(0, 0, 0, 0);
      v[i][0] = a.x; v[i][1] = a.y; v[i][2] = a.z; v[i][3] = a.w;
      v[i][4] = b.x; v[i][5] = b.y; v[i][6] = b.z; v[i][7] = b.w;
    }
    auto row_rinv = [&]() {  // 1 / rms of the row held in v (block-wide)
      double ss = 0.0;
#pragma unroll
      for (int i = 0; i < kHeld; ++i)
#pragma unroll
        for (int e = 0; e < 8; ++e) ss += (double)v[i][e] * v[i][e];
      ss = warp_sum(ss);
      if (lane == 0) red[warp] = ss;
      __syncthreads();
      ss = 0.0;
#pragma unroll
      for (int i = 0; i < 8; ++i) ss += red[i];
      __syncthreads();  // red may be written again
      return (float)(1.0 / sqrt(ss / (double)K + (double)p.eps));
    };
    if (p.gamma) {
      const float rinv = row_rinv();
#pragma unroll
      for (int i = 0; i < kHeld; ++i) {
        const int k = tid * 8 + i * 2048;
        if (k >= K) continue;
        const float4 ga = __ldg(reinterpret_cast<const float4*>(p.gamma + k));
        const float4 gb = __ldg(reinterpret_cast<const float4*>(p.gamma + k + 4));
        const float g[8] = {ga.x, ga.y, ga.z, ga.w, gb.x, gb.y, gb.z, gb.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) v[i][e] = __fmul_rn(__fmul_rn(v[i][e], rinv), g[e]);
      }
    }
    if (p.rowscale) {
      float amax = 0.f;
#pragma unroll
      for (int i = 0; i < kHeld; ++i)
#pragma unroll
        for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(v[i][e]));  // rows past K hold zeros
      inv_s = row_scale(amax);
    }
#pragma unroll
    for (int i = 0; i < kHeld; ++i) {
      const int k = tid * 8 + i * 2048;
      if (k < K) emit(k, v[i]);
    }
    return;
  }
  float rinv = 1.f;
  if (p.gamma) {
    double ss = 0.0;
    for (int k = tid; k < K; k += 256) {
      const float v = xg[k];
      ss += (double)v * v;
    }
    ss = warp_sum(ss);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    ss = 0.0;
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += red[i];
    rinv = (float)(1.0 / sqrt(ss / (double)K + (double)p.eps));
  }
  if (p.rowscale) {
    float amax = 0.f;
    for (int k = tid; k < K; k += 256)
      amax = fmaxf(amax, fabsf(p.gamma ? __fmul_rn(__fmul_rn(xg[k], rinv), p.gamma[k]) : xg[k]));
    inv_s = row_scale(amax);
  }
  for (int k = tid * 8; k < K; k += 256 * 8) {
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e)
      v[e] = p.gamma ? __fmul_rn(__fmul_rn(xg[k + e], rinv), p.gamma[k + e]) : xg[k + e];
    emit(k, v);
  }
}

// kind::f16 with both operands through shared-memory descriptors, for a converged warp: every lane
// calls, one issues.
__device__ __forceinline__ void lm_umma_f16_w(uint32_t tmem_d, uint32_t alo, uint32_t blo, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t.reg .b64 ad, bd;\n\tmov.b64 ad, {%1, %5};\n\tmov.b64 bd, {%2, %6};\n\t"
      "elect.sync _|e, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], ad, bd, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(alo), "r"(blo), "r"(idesc), "r"(accumulate), "n"(tc_desc_hi(1024) | (2u << 29)), "n"(tc_desc_hi(1024))
      : "memory");
}

template <int TS>
__global__ void __launch_bounds__(kLmThreads, 1) lmhead_mma_kernel(const __grid_constant__ LmMmaParams p) {
  using Cfg = LmCfg<TS>;
  constexpr int kAS = Cfg::kAStages, kBS = Cfg::kBStages, kN = Cfg::kN;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int nblk = p.K / kLmBlock, nsteps = (nblk + 1) / 2;  // the last step may hold one block
  const int t0 = (int)((long)p.ntiles * blockIdx.x / gridDim.x);
  const int t1 = (int)((long)p.ntiles * (blockIdx.x + 1) / gridDim.x);

  uint64_t* a_full = reinterpret_cast<uint64_t*>(smem);  // [kAS] table boxes landed
  uint64_t* a_free = a_full + kAS;                        // [kAS] their MMAs have retired
  uint64_t* b_full = a_free + kAS;                        // [kBS] activations landed
  uint64_t* b_free = b_full + kBS;                        // [kBS]
  uint64_t* acc_full = b_free + kBS;                      // a round's products are complete
  uint64_t* acc_free = acc_full + 1;                      // the epilogue has read them
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + 1);
  unsigned long long* wkeys = reinterpret_cast<unsigned long long*>(smem + 1024);  // [16][TS]
  uint8_t* astg = smem + Cfg::kCtrl;
  uint8_t* bstg = astg + kAS * kLmABytes;

  if (tid == 0) {
    for (int i = 0; i < kAS; ++i) {
      mbar_init(&a_full[i], 1);
      mbar_init(&a_free[i], 1);
    }
    for (int i = 0; i < kBS; ++i) {
      mbar_init(&b_full[i], 1);
      mbar_init(&b_free[i], 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_free, kLmEpiWarps);
    fence_mbar_init();
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
        smem_u32(tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_before_sync();
  __syncthreads();
  tc_after_sync();
  constexpr uint32_t tmem = 0;  // all 512 columns are this CTA's
  bool ok = true;
  pdl_trigger();

  if (warp == 0) {
    // ================= table: constant, so no wait on the previous kernel =======================
    const uint64_t pol = policy_evict_first();
    TcRing<kAS> r;
    int nth = 0;
    for (int t = t0; t < t1 && ok; t += Cfg::kTiles) {
      const int n = min(Cfg::kTiles, t1 - t);
      for (int ks = 0; ks < nsteps && ok; ++ks)
        for (int i = 0; i < n; ++i, r.advance()) {
          if (nth++ == kAS) pdl_wait();  // from here on a slot is freed by a product (bounded waits)
          ok = tc_wait_w(&a_free[r.i], r.phase ^ 1, p.status);
          if (!ok) break;
          if (tc_elect()) {
            const int nb = min(2, nblk - 2 * ks);
            mbar_arrive_expect_tx(&a_full[r.i], nb * kLmABox);
            for (int h = 0; h < nb; ++h)
              tc_tma_box_2d(astg + (size_t)r.i * kLmABytes + h * kLmABox, &p.tmap, (2 * ks + h) * kLmBlock,
                            (t + i) * kLmRows, &a_full[r.i], pol);
          }
          __syncwarp();
        }
    }
  } else if (warp == 1) {
    // ================= activations: written by the kernel before this one =======================
    pdl_wait();
    TcRing<kBS> r;
    for (int t = t0; t < t1 && ok; t += Cfg::kTiles)
      for (int ks = 0; ks < nsteps; ++ks, r.advance()) {
        ok = tc_wait_w(&b_free[r.i], r.phase ^ 1, p.status);
        if (!ok) break;
        if (tc_elect()) {
          const uint32_t bytes = (uint32_t)min(2, nblk - 2 * ks) * Cfg::kBBlock;
          mbar_arrive_expect_tx(&b_full[r.i], bytes);
          bulk_g2s(bstg + (size_t)r.i * Cfg::kBBytes, p.xb + (size_t)ks * Cfg::kBBytes, bytes, &b_full[r.i]);
        }
        __syncwarp();
      }
  } else if (warp == 2) {
    // ================= MMA issue: the whole warp runs the loop, one lane issues =================
    // Control flow does not depend on a wait's outcome (ring positions stay provably uniform);
    // after an expired wait the products run on whatever is there, the status word says so.
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      if (!mbar_try_wait(bar, parity) && ok) ok = tc_wait_slow(smem_u32(bar), parity, p.status);
    };
    pdl_wait();  // so that the first wait below is bounded by this kernel's own copies
    TcRing<kAS> ra;
    TcRing<kBS> rb;
    const uint32_t a0 = tc_desc_lo(smem_u32(astg), 0), b0 = tc_desc_lo(smem_u32(bstg), 128);
    uint32_t phase = 1;
    for (int t = t0; t < t1; t += Cfg::kTiles, phase ^= 1) {
      const int n = min(Cfg::kTiles, t1 - t);
      wait(acc_free, phase);
      for (int ks = 0; ks < nsteps; ++ks, rb.advance()) {
        wait(&b_full[rb.i], rb.phase);
        const uint32_t bd = b0 + rb.i * (Cfg::kBBytes >> 4);
        for (int i = 0; i < n; ++i, ra.advance()) {
          wait(&a_full[ra.i], ra.phase);
          tc_after_sync();
          const uint32_t ad = a0 + ra.i * (kLmABytes >> 4);
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (2 * ks + h < nblk) {
#pragma unroll
              for (int j = 0; j < kLmBlock / 16; ++j)  // K = 16 elements = 32 bytes per instruction
                lm_umma_f16_w(tmem + i * kN, ad + h * (kLmABox >> 4) + j * 2, bd + h * (Cfg::kBBlock >> 4) + j * 16,
                              p.idesc, (ks > 0 || h > 0 || j > 0) ? 1u : 0u);
            }
          tc_commit_w(&a_free[ra.i]);
        }
        tc_commit_w(&b_free[rb.i]);
      }
      tc_commit_w(acc_full);
    }
  } else if (warp >= 4) {
    // ================= epilogue ==================================================================
    const int q = warp & 3, s4 = (warp >> 2) - 1;  // lane quarter, which accumulators
    pdl_wait();  // the row scales; logits and keys may still be in use before this
    unsigned long long best[TS / 16];  // lane e < 16: key of token 16 c + e over this warp's rows
    float rs[TS / 16];                 // and that token's row scale, handed around by shuffles
#pragma unroll
    for (int c = 0; c < TS / 16; ++c) {
      const int m = 16 * c + (lane & 15);
      best[c] = 0ull;
      rs[c] = p.rowscale && m < p.M ? __ldcg(p.rowscale + m) : 1.f;
    }
    uint32_t phase = 0;
    for (int t = t0; t < t1; t += Cfg::kTiles, phase ^= 1) {
      const int n = min(Cfg::kTiles, t1 - t);
      ok = ok && tc_wait_w(acc_full, phase, p.status);
      tc_after_sync();
      for (int i = s4; i < n; i += 4) {
        const long row = (long)(t + i) * kLmRows + q * 32 + lane;
        const bool row_ok = row < p.V;
        const uint32_t addr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(i * kN);
#pragma unroll
        for (int c = 0; c < TS / 16; ++c) {
          if (c * 16 >= p.M) break;  // the same for the whole warp
          uint32_t hi[16], lo[16];
          HB_TMEM_LD16(hi, addr + 16 * c);
          HB_TMEM_LD16(lo, addr + TS + 16 * c);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const int m = 16 * c + e;
            float v = __fadd_rn(__uint_as_float(hi[e]), __uint_as_float(lo[e]));
            v *= __shfl_sync(0xffffffffu, rs[c], e);  // undo the staging's row scale (exact)
            if (m < p.M && row_ok && p.logits && ok) p.logits[(size_t)m * p.V + row] = v;
            if (!p.keys) continue;
            uint32_t u = __float_as_uint(v);
            u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);  // monotone map float -> uint
            if (!(v == v) || !row_ok) u = 0u;                  // NaN and padding rows never win
            const uint32_t top = __reduce_max_sync(0xffffffffu, u);
            const uint32_t who = __ballot_sync(0xffffffffu, u == top);
            if (lane == e && top) {
              const uint32_t first = (uint32_t)(row - lane) + (uint32_t)(__ffs(who) - 1);
              const unsigned long long k =
                  ((unsigned long long)top << 32) | (unsigned long long)(0xFFFFFFFFu - first);
              best[c] = k > best[c] ? k : best[c];
            }
          }
        }
      }
      tc_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_free);
    }
    if (p.keys) {
#pragma unroll
      for (int c = 0; c < TS / 16; ++c)
        if (lane < 16) wkeys[(warp - 4) * TS + 16 * c + lane] = best[c];
      asm volatile("bar.sync 1, %0;" ::"n"(kLmEpiWarps * 32) : "memory");
      const int m = tid - 128;
      if (m < p.M && ok) {
        unsigned long long k = wkeys[m];
#pragma unroll
        for (int w = 1; w < kLmEpiWarps; ++w) {
          const unsigned long long o = wkeys[w * TS + m];
          k = o > k ? o : k;
        }
        if (k) atomicMax(&p.keys[m], k);
      }
    }
  }
  tc_before_sync();
  __syncthreads();
  if (warp == 2)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(*tmem_slot));
}

}  // namespace hb

using namespace hb;

template <int TS>
static int lm_launch(hb200_ctx* ctx, LmMmaParams& p, int dtype, cudaStream_t st) {
  using Cfg = LmCfg<TS>;
  // instruction descriptor of kind::f16: D = f32, A and B of the table's type, both K-major
  const uint32_t fmt = dtype == 0 ? 1u : 0u;  // 1 = bf16, 0 = f16
  p.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(Cfg::kN >> 3) << 17) |
            ((uint32_t)(kLmRows >> 4) << 24);
  const int rc = hb_func_smem(ctx, reinterpret_cast<const void*>(lmhead_mma_kernel<TS>), (size_t)Cfg::kSmem);
  if (rc != HB200_OK) return rc;
  const int grid = p.ntiles < ctx->sm_count ? p.ntiles : ctx->sm_count;
  HB_CUDA(launch_pdl(lmhead_mma_kernel<TS>, dim3((unsigned)grid), dim3(kLmThreads), (size_t)Cfg::kSmem, st,
                     ctx->pdl, p));
  return HB200_OK;
}

// Batched LM head (16 <= M <= 64, K a multiple of 64): logits (nullable) and argmax keys (atomicMax
// like the batch-1 LM head, so that the finishing kernel is shared).
int hb_lmhead_mma_run(hb200_ctx* ctx, const void* d_table, int dtype, long V, int K,
                      const float* d_x, int M, const float* d_rms_gamma, float rms_eps,
                      float* d_logits, unsigned long long* d_keys, cudaStream_t st) {
  ScratchUse use(ctx, st);  // the staged hi / lo activations
  HB_REQUIRE(V >= 1 && V < (1l << 31), "lmhead (batched): bad row count");
  HB_REQUIRE(M >= 1 && M <= 64, "lmhead (batched): M=%d", M);
  const int slots = M <= 32 ? 32 : 64;
  const size_t xb_bytes = (size_t)(K / kLmBlock) * slots * 256;
  HB_REQUIRE(kScratchLmSplit + xb_bytes <= kScratchSplitK,
             "lmhead (batched): K=%d needs %zu bytes of activation scratch", K, xb_bytes);
  uint8_t* xb = static_cast<uint8_t*>(ctx->d_scratch) + kScratchLmSplit;
  // bf16 has the exponent range of f32.  At the start of the scratch: the blocks may fill the region
  // in front of the split-K partials to its end
  float* rowscale = dtype == 1 ? static_cast<float*>(ctx->d_scratch) : nullptr;
  LmMmaParams p = {};
  TcEncodeTiledFn encode = tc_tensor_map_encoder();
  HB_REQUIRE(encode != nullptr, "lmhead (batched): the driver has no cuTensorMapEncodeTiled");
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)V};
  const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kLmBlock, (cuuint32_t)kLmRows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult erc =
      encode(&p.tmap, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(d_table), dims, strides,
             box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  HB_REQUIRE(erc == CUDA_SUCCESS, "lmhead (batched): cuTensorMapEncodeTiled failed (%d)", (int)erc);
  const LmSplitParams sp = {d_x, d_rms_gamma, rms_eps, K, M, dtype, slots, xb, rowscale};
  HB_CUDA(launch_pdl(lm_split_kernel, dim3(slots), dim3(256), 0, st, ctx->pdl, sp));
  p.xb = xb;
  p.logits = d_logits;
  p.keys = d_keys;
  p.V = V;
  p.K = K;
  p.M = M;
  p.ntiles = (int)((V + kLmRows - 1) / kLmRows);
  p.rowscale = rowscale;
  p.status = ctx->d_status;
  return slots == 32 ? lm_launch<32>(ctx, p, dtype, st) : lm_launch<64>(ctx, p, dtype, st);
}
