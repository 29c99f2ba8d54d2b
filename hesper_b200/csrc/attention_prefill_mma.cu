// attention_prefill_mma.cu -- causal GQA attention of a short prompt chunk on mma.sync: the kernel that
// attention_prefill.cu hands the shapes to whose few tiles do not pay for the tensor-memory
// pipeline (its pf_use_mma says which, with both sides' times).
//
// A CTA owns 64 query rows -- 64 / G consecutive tokens times the G query heads of one KV head -- and
// walks the positions those tokens see in tiles of 64 (32 at head_dim 256):
//   * Q (pre-multiplied by scale * log2 e, f16) stays in shared memory for the whole CTA;
//   * K/V tiles arrive by 16-byte cp.async into a two-stage ring (XOR-swizzled 16-byte units,
//     conflict-free ldmatrix); ring caches map position p to slot p % slots;
//   * S = Q K^T and O += P V on mma.sync.m16n8k16 (f16 in, f32 accumulate), one warp per 16 rows;
//     the softmax is the online form in the exp2 domain, P is rounded to f16 for the second
//     product (same rounding as the decode kernel's FAST mode: bar 2e-3 against an f64 evaluation);
//   * a row's visible positions are [max(0, pos - window + 1), pos] with pos the token's own
//     position: causal inside the chunk, sliding window if asked.
// What bounds it: latency.  A chunk of 8 tokens over 16 positions takes 4.8 us at head_dim 64 where
// the tcgen05 kernel takes 6.7 (allocation, barriers, two hops through tensor memory), a 64-position
// tile about 1.2 us in either; several of these CTAs share an SM, one of the other does not.
#include <math_constants.h>

#include "attention_prefill.cuh"

namespace hb {

constexpr int kPmWarps = 4;
constexpr int kPmThreads = kPmWarps * 32;
// positions per K/V tile: 64, and 32 at head_dim 256, where the 128 output accumulators per
// lane leave no registers for a 64-wide score tile
template <int D>
struct PmTile {
  static constexpr int value = D >= 256 ? 32 : 64;
};

template <int D>
struct PmCfg {
  static constexpr int kQStride = D + 8;                      // halves per Q row (bank spread)
  static constexpr int kQBytes = kPmRows * kQStride * 2;
  static constexpr int kRowBytes = D * 2;
  static constexpr int kTile = PmTile<D>::value;
  static constexpr int kTileBytes = kTile * kRowBytes;        // one of K or V
  static constexpr int kSmem = kQBytes + 2 * 2 * kTileBytes;  // Q + two stages of (K, V)
};

__device__ __forceinline__ void pm_cp16(void* dst, const void* src, bool valid) {
  const uint32_t n = valid ? 16u : 0u;  // src-size 0: the 16 bytes are zero-filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(n)
               : "memory");
}
__device__ __forceinline__ void pm_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void pm_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void pm_ldsm(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_u32(p)));
}
__device__ __forceinline__ void pm_ldsm_t(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_u32(p)));
}
__device__ __forceinline__ void pm_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                       uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pm_pack(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

template <int D>
__global__ void __launch_bounds__(kPmThreads, D >= 256 ? 1 : 2)
    attn_prefill_mma_kernel(const __grid_constant__ PmParams p) {
  using Cfg = PmCfg<D>;
  constexpr int KS = D / 16;  // k-steps of the first product
  constexpr int NO = D / 8;   // n-tiles of the output
  constexpr int CPR = D / 8;  // 16-byte units per cache row
  constexpr int TILE = Cfg::kTile, NS = TILE / 8;  // positions and score n-tiles per K/V tile
  extern __shared__ __align__(128) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int G = p.G, TQ = kPmRows / G;
  const int qt = blockIdx.x / p.nsplit, split = blockIdx.x % p.nsplit;
  const int kvh = blockIdx.y, b = blockIdx.z;

  __half* qs = reinterpret_cast<__half*>(smem);
  uint8_t* stage0 = smem + Cfg::kQBytes;

  pdl_trigger();
  pdl_wait();  // q, the cache rows of this chunk and seqlens come from earlier kernels

  int len = max(p.seqlens[b], 0);  // positions after the chunk
  if (!p.ring) len = min(len, p.slots);  // a corrupt length never overruns a linear cache
  const int t0 = qt * TQ;                // first token of this CTA
  const int t1 = min(t0 + TQ, p.T) - 1;  // last one
  // positions of the chunk's tokens: token t sits at len - T + t
  const int pos_first = len - p.T + t0, pos_last = len - p.T + t1;
  int kv_lo = 0;
  if (p.window > 0) kv_lo = max(0, pos_first - p.window + 1);
  const int kv_hi = pos_last;  // inclusive
  const int ntiles_all = kv_hi >= kv_lo ? (kv_hi - kv_lo) / TILE + 1 : 0;
  // this CTA's share of the tiles
  const int tps = (ntiles_all + p.nsplit - 1) / p.nsplit;
  const int j0 = split * tps;
  const int ntiles = max(0, min(ntiles_all, j0 + tps) - j0);

  const __half* kbase = p.k + ((size_t)b * p.Hkv + kvh) * (size_t)p.slots * D;
  const __half* vbase = p.v + ((size_t)b * p.Hkv + kvh) * (size_t)p.slots * D;
  auto issue = [&](int j, int st) {
    uint8_t* ks = stage0 + (size_t)st * 2 * Cfg::kTileBytes;
    uint8_t* vs = ks + Cfg::kTileBytes;
    const int p0 = kv_lo + (j0 + j) * TILE;
#pragma unroll
    for (int i = 0; i < TILE * CPR / kPmThreads; ++i) {
      const int u = tid + i * kPmThreads;
      const int row = u / CPR, cc = u % CPR;
      const int pos = p0 + row;
      const bool ok = pos <= kv_hi && pos >= 0;
      int slot = ok ? pos : 0;
      if (p.ring) slot %= p.slots;
      const size_t goff = (size_t)slot * D + cc * 8;
      const int soff = row * Cfg::kRowBytes + ((cc ^ (row & 7)) << 4);
      pm_cp16(ks + soff, kbase + goff, ok);
      pm_cp16(vs + soff, vbase + goff, ok);
    }
  };
  if (ntiles > 0) issue(0, 0);
  pm_commit();

  // Q rows: row r = (token t0 + r / G, head kvh * G + r % G), scaled, f16; rows past T are zero
  for (int i = tid; i < kPmRows * (D / 4); i += kPmThreads) {
    const int r = i / (D / 4), d4 = i % (D / 4);
    const int t = t0 + r / G, h = kvh * G + r % G;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < p.T) {
      const size_t qi = (((size_t)b * p.T + t) * p.H + h) * D + 4 * d4;
      if (p.q_is_f16) {
        const __half2* hq = reinterpret_cast<const __half2*>(reinterpret_cast<const __half*>(p.q) + qi);
        const float2 a = __half22float2(hq[0]), c = __half22float2(hq[1]);
        v = make_float4(a.x, a.y, c.x, c.y);
      } else {
        v = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.q) + qi);
      }
    }
    uint2 w;
    w.x = pm_pack(v.x * p.scale_log2, v.y * p.scale_log2);
    w.y = pm_pack(v.z * p.scale_log2, v.w * p.scale_log2);
    *reinterpret_cast<uint2*>(qs + r * Cfg::kQStride + 4 * d4) = w;
  }
  __syncthreads();

  // this lane's two rows (g and g + 8 of the warp's 16) and what they may see
  const int rA = 16 * warp + g, rB = rA + 8;
  const int tA = t0 + rA / G, tB = t0 + rB / G;
  const int posA = len - p.T + tA, posB = len - p.T + tB;
  const int loA = p.window > 0 ? max(0, posA - p.window + 1) : 0;
  const int loB = p.window > 0 ? max(0, posB - p.window + 1) : 0;
  const bool liveA = tA < p.T, liveB = tB < p.T;

  float mA = -CUDART_INF_F, mB = -CUDART_INF_F, lA = 0.f, lB = 0.f;
  float o[NO][4];
#pragma unroll
  for (int n = 0; n < NO; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;

  for (int j = 0; j < ntiles; ++j) {
    if (j + 1 < ntiles) issue(j + 1, (j + 1) & 1);
    pm_commit();
    pm_wait<1>();
    __syncthreads();  // tile j is in shared memory for every warp
    const uint8_t* ks = stage0 + (size_t)(j & 1) * 2 * Cfg::kTileBytes;
    const uint8_t* vs = ks + Cfg::kTileBytes;
    const int p0 = kv_lo + (j0 + j) * TILE;

    // ---- S = Q K^T: 16 rows x TILE positions per warp -------------------------------------
    float s[NS][4];
#pragma unroll
    for (int n = 0; n < NS; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
    for (int kk = 0; kk < KS; ++kk) {
      uint32_t a[4];
      {
        // A fragment of Q: matrices (rows 0-7 | 8-15) x (k 0-7 | 8-15) of this warp's 16 rows
        const int row = 16 * warp + (lane & 7) + ((lane >> 3) & 1) * 8;
        const int col = 16 * kk + (lane >> 4) * 8;
        pm_ldsm(a, qs + row * Cfg::kQStride + col);
      }
#pragma unroll
      for (int np = 0; np < NS / 2; ++np) {  // two n-tiles (16 positions) per ldmatrix
        uint32_t kb[4];
        // matrices: (pos 0-7, d 0-7), (pos 0-7, d 8-15), (pos 8-15, d 0-7), (pos 8-15, d 8-15)
        const int row = 16 * np + (lane & 7) + (lane >> 4) * 8;
        const int cc = 2 * kk + ((lane >> 3) & 1);
        pm_ldsm(kb, ks + row * Cfg::kRowBytes + ((cc ^ (row & 7)) << 4));
        pm_mma(s[2 * np], a, kb[0], kb[1]);
        pm_mma(s[2 * np + 1], a, kb[2], kb[3]);
      }
    }

    // ---- mask, online softmax (exp2 domain) ----------------------------------------------
    float mxA = -CUDART_INF_F, mxB = -CUDART_INF_F;
#pragma unroll
    for (int n = 0; n < NS; ++n) {
      const int pc = p0 + 8 * n + 2 * t4;
      const bool a0 = liveA && pc >= loA && pc <= posA, a1 = liveA && pc + 1 >= loA && pc + 1 <= posA;
      const bool b0 = liveB && pc >= loB && pc <= posB, b1 = liveB && pc + 1 >= loB && pc + 1 <= posB;
      s[n][0] = a0 ? s[n][0] : -CUDART_INF_F;
      s[n][1] = a1 ? s[n][1] : -CUDART_INF_F;
      s[n][2] = b0 ? s[n][2] : -CUDART_INF_F;
      s[n][3] = b1 ? s[n][3] : -CUDART_INF_F;
      mxA = fmaxf(mxA, fmaxf(s[n][0], s[n][1]));
      mxB = fmaxf(mxB, fmaxf(s[n][2], s[n][3]));
    }
    mxA = fmaxf(mxA, __shfl_xor_sync(0xffffffffu, mxA, 1));
    mxA = fmaxf(mxA, __shfl_xor_sync(0xffffffffu, mxA, 2));
    mxB = fmaxf(mxB, __shfl_xor_sync(0xffffffffu, mxB, 1));
    mxB = fmaxf(mxB, __shfl_xor_sync(0xffffffffu, mxB, 2));
    const float mnA = fmaxf(mA, mxA), mnB = fmaxf(mB, mxB);
    const float baseA = mnA == -CUDART_INF_F ? 0.f : mnA;  // nothing visible yet: avoid inf - inf
    const float baseB = mnB == -CUDART_INF_F ? 0.f : mnB;
    const float alA = exp2f(mA - baseA), alB = exp2f(mB - baseB);
    float sumA = 0.f, sumB = 0.f;
    uint32_t pa[NS / 2][4];  // P as A fragments of the second product: k-steps of 16 positions
#pragma unroll
    for (int n = 0; n < NS; ++n) {
      const float e0 = exp2f(s[n][0] - baseA), e1 = exp2f(s[n][1] - baseA);
      const float e2 = exp2f(s[n][2] - baseB), e3 = exp2f(s[n][3] - baseB);
      sumA += e0 + e1;
      sumB += e2 + e3;
      pa[n >> 1][(n & 1) * 2] = pm_pack(e0, e1);      // rows g
      pa[n >> 1][(n & 1) * 2 + 1] = pm_pack(e2, e3);  // rows g + 8
    }
    sumA += __shfl_xor_sync(0xffffffffu, sumA, 1);
    sumA += __shfl_xor_sync(0xffffffffu, sumA, 2);
    sumB += __shfl_xor_sync(0xffffffffu, sumB, 1);
    sumB += __shfl_xor_sync(0xffffffffu, sumB, 2);
    lA = lA * alA + sumA;
    lB = lB * alB + sumB;
    mA = mnA;
    mB = mnB;
#pragma unroll
    for (int n = 0; n < NO; ++n) {
      o[n][0] *= alA;
      o[n][1] *= alA;
      o[n][2] *= alB;
      o[n][3] *= alB;
    }

    // ---- O += P V ---------------------------------------------------------------------------
#pragma unroll
    for (int kk = 0; kk < NS / 2; ++kk) {  // 16 positions per step
#pragma unroll
      for (int np = 0; np < NO / 2; ++np) {  // two n-tiles (16 dims) per ldmatrix
        uint32_t vb[4];
        // transposed matrices: (pos 0-7 | 8-15) x (d 0-7 | 8-15) of this step
        const int row = 16 * kk + (lane & 7) + ((lane >> 3) & 1) * 8;
        const int cc = 2 * np + (lane >> 4);
        pm_ldsm_t(vb, vs + row * Cfg::kRowBytes + ((cc ^ (row & 7)) << 4));
        pm_mma(o[2 * np], pa[kk], vb[0], vb[1]);
        pm_mma(o[2 * np + 1], pa[kk], vb[2], vb[3]);
      }
    }
    __syncthreads();  // every warp is done with stage j & 1 before it is refilled
  }

  // ---- normalise and store, or hand the partial to the merge kernel ------------------------
  if (p.nsplit == 1) {
    const float invA = lA > 0.f ? 1.f / lA : 0.f, invB = lB > 0.f ? 1.f / lB : 0.f;
    if (liveA) {
      float* dst = p.out + (((size_t)b * p.T + tA) * p.H + kvh * G + rA % G) * D;
#pragma unroll
      for (int n = 0; n < NO; ++n)
        *reinterpret_cast<float2*>(dst + 8 * n + 2 * t4) = make_float2(o[n][0] * invA, o[n][1] * invA);
    }
    if (liveB) {
      float* dst = p.out + (((size_t)b * p.T + tB) * p.H + kvh * G + rB % G) * D;
#pragma unroll
      for (int n = 0; n < NO; ++n)
        *reinterpret_cast<float2*>(dst + 8 * n + 2 * t4) = make_float2(o[n][2] * invB, o[n][3] * invB);
    }
    return;
  }
  if (liveA) {
    const size_t pi = ((((size_t)b * p.T + tA) * p.H + kvh * G + rA % G) * p.nsplit + split);
    float* dst = p.part_o + pi * D;
#pragma unroll
    for (int n = 0; n < NO; ++n)
      *reinterpret_cast<float2*>(dst + 8 * n + 2 * t4) = make_float2(o[n][0], o[n][1]);
    if (t4 == 0) *reinterpret_cast<float2*>(p.part_ml + pi * 2) = make_float2(mA, lA);
  }
  if (liveB) {
    const size_t pi = ((((size_t)b * p.T + tB) * p.H + kvh * G + rB % G) * p.nsplit + split);
    float* dst = p.part_o + pi * D;
#pragma unroll
    for (int n = 0; n < NO; ++n)
      *reinterpret_cast<float2*>(dst + 8 * n + 2 * t4) = make_float2(o[n][2], o[n][3]);
    if (t4 == 0) *reinterpret_cast<float2*>(p.part_ml + pi * 2) = make_float2(mB, lB);
  }
}

}  // namespace hb

using namespace hb;

// How many CTAs share the K/V range of a query tile: 1 when the query tiles alone fill the SMs,
// else enough to, but no split shorter than 4 tiles of the longest range a tile can see and
// at most 8.  A function of the shapes only (the workspace is sized with it).
int hb_attn_prefill_mma_splits(const hb200_ctx* ctx, int nseq, int T, int G, int Hkv, int D, long span) {
  const int TQ = kPmRows / G;
  const long ctas = (long)((T + TQ - 1) / TQ) * Hkv * nseq;
  if (ctas >= ctx->sm_count) return 1;
  const int tile = D >= 256 ? 32 : 64;
  const long most = (span + tile - 1) / tile / 4;
  long ns = (ctx->sm_count + ctas - 1) / ctas;
  if (ns > 8) ns = 8;
  if (ns > most) ns = most;
  return ns < 1 ? 1 : (int)ns;
}

template <int D>
static int pm_launch(hb200_ctx* ctx, const PmParams& p, cudaStream_t st) {
  const int rc = hb_func_smem(ctx, reinterpret_cast<const void*>(attn_prefill_mma_kernel<D>), PmCfg<D>::kSmem);
  if (rc) return rc;
  const int TQ = kPmRows / p.G;
  const dim3 grid((unsigned)((p.T + TQ - 1) / TQ) * p.nsplit, (unsigned)p.Hkv, (unsigned)p.nseq);
  HB_CUDA(launch_pdl(attn_prefill_mma_kernel<D>, grid, dim3(kPmThreads), (size_t)PmCfg<D>::kSmem, st, ctx->pdl, p));
  return HB200_OK;
}

int hb_attn_prefill_mma(hb200_ctx* ctx, const PmParams& p, int D, cudaStream_t st) {
  switch (D) {
    case 64: return pm_launch<64>(ctx, p, st);
    case 128: return pm_launch<128>(ctx, p, st);
    default: return pm_launch<256>(ctx, p, st);
  }
}
