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
// What bounds it: at 64 tokens the dequantiser (about 3 instructions per weight) and HBM, at
// 256 tokens the tensor pipe (M=128, N=256, K=16 in 138 cycles).  Either way only when every SM
// works, so the work is dealt in units of (row tile of 128, super-block of 256 weights):
//   * whole waves of row tiles go one tile to a CTA (W per CTA, results stored directly);
//   * the R row tiles left over are cut along K into runs of `upc` consecutive units, one run
//     per CTA.  A run that does not cover its tile leaves an f32 partial in the context's
//     scratch and a small second kernel adds a tile's partials in K order (deterministic).
//     160 tiles of a 10240-row gate/up pair so take 11 super-block times on 148 SMs instead of
//     20, the 20 tiles of a 2560-row down projection 6 instead of 40.
// 19 warps with fixed roles:
//   warps 0-15 dequantise: warps 0-7 the even, 8-15 the odd steps of 128 weights; a thread owns
//              one row and 64 weights of a step and stores them with one tcgen05.st.  They also
//              run the epilogue of a finished tile, after they have refilled the A stages for
//              the next one;
//   warp 16    weights: 2-D tensor-map TMA boxes of 64 rows x 256 weights, a ring of 2 to 7 tiles;
//   warp 17    activations: bulk copies of the step's tiles (f16, operand layout written by the
//              staging kernel);
//   warp 18    one elected thread issues the MMAs (M=128, N=NT tokens, K=16).
// A gate/up pair is one launch: a tile holds 64 gate rows and the 64 up rows of the same outputs,
// dealt to the tensor-memory lanes so that a gate lane's up value sits 16 lanes further in the
// same warp (one shuffle per two tokens in the epilogue).
// Every wait is bounded; on expiry the kernel still releases its tensor memory.
#include <cuda_fp16.h>

#include "tcgen05.cuh"

namespace hb {

constexpr int kQmRows = 128;          // weight rows per tile = MMA M
constexpr int kQmStepK = 128;         // weights per pipeline step (half a super-block)
constexpr int kQmACols = kQmStepK / 2;  // 64 TMEM columns of f16 pairs per stage
constexpr int kQmExpWarps = 16;
constexpr int kQmThreads = (kQmExpWarps + 3) * 32;
constexpr int kQmMaxSeg = 4;          // tensors one launch multiplies by the same activations

// NT tokens per pass = MMA N; a unit is the bytes of 256 weights (one Q4_K super-block, eight
// Q8_0 blocks).
template <int NT, int FMT>
struct QmCfg {
  static constexpr int kUnit = FMT == 12 ? 144 : 272;
  static constexpr int kPkBytes = kQmRows * kUnit;          // 18 / 34 KB
  static constexpr int kAccBufs = NT <= 128 ? 2 : 1;        // accumulators in tensor memory
  static constexpr int kA0 = kAccBufs * NT;                 // first TMEM column of the A stages
  static constexpr int kAStages = NT == 64 ? 6 : 4;
  // activation stages: a whole step, or half of one at 256 tokens (64 KB per step)
  static constexpr int kBPer = NT == 256 ? 2 : 1;
  static constexpr int kBBytes = NT * kQmStepK * 2 / kBPer;  // 16 / 32 / 32 KB
  static constexpr int kBStages = NT == 64 ? 6 : 4;
  static constexpr int kPkStages = FMT == 12 ? (NT == 64 ? 7 : 5) : (NT == 64 ? 3 : 2);
  static constexpr int kSmem = 1024 + kPkStages * kPkBytes + kBStages * kBBytes;
  static_assert(kA0 + kAStages * kQmACols <= 512, "tensor memory columns");
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
  const uint8_t* xb;      // f16 activations: [K/64][NT rows x 64 f16, operand layout]
  const float* rowscale;  // [NT] power of two each token's row was divided by before rounding
  int M;
  float* part;            // [cta][2][NT tokens][128 lanes] partial sums of left-over tiles
  uint32_t idesc;
  uint32_t* status;
};

// 0.5*g*(1+tanh(sqrt(2/pi)*(g+0.044715 g^3))), the gate factor of the GeGLU
// (Hesper/Layers/FusedFFNSpec.lean:42-45), same expression as the standalone kernel
__device__ __forceinline__ float glu_gate(float g) {
  const float t = 0.7978845608028654f * (g + 0.044715f * g * g * g);
  return 0.5f * g * (1.0f + tanhf(t));
}

__device__ __forceinline__ uint32_t pack_f16(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float2 h2f(uint32_t h) {
  return __half22float2(*reinterpret_cast<const __half2*>(&h));
}
// {a.x*s + c, a.y*s + c} in one packed instruction
__device__ __forceinline__ float2 fma2(float2 a, float2 s, float2 c) {
  float2 r;
  asm("{\n\t.reg .b64 a, s, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 s, {%4, %5};\n\t"
      "mov.b64 c, {%6, %7};\n\tfma.rn.f32x2 d, a, s, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(s.x), "f"(s.y), "f"(c.x), "f"(c.y));
  return r;
}

// 32 nibble bytes of a chunk (two sub-blocks of 32 weights: low and high nibbles) -> 64 f16 as
// fma(ds, q, -dm) in f32, rounded once.  A nibble is moved to bits 4-7 of a 16-bit lane and
// completed to the f16 1024 + 16 q with one LOP3 for two of them; widened exactly, the f32 fma
// takes scale ds / 16 and addend -dm - 64 ds.  o[0..15]: low, o[16..31]: high nibbles.
__device__ __forceinline__ void q4k_expand(const uint32_t (&q)[8], float ds0, float dm0, float ds1,
                                           float dm1, uint32_t (&o)[32]) {
  const float2 s0 = make_float2(ds0 * 0.0625f, ds0 * 0.0625f);
  const float2 s1 = make_float2(ds1 * 0.0625f, ds1 * 0.0625f);
  const float a0 = fmaf(-64.f, ds0, -dm0), a1 = fmaf(-64.f, ds1, -dm1);
  const float2 c0 = make_float2(a0, a0), c1 = make_float2(a1, a1);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t w = q[i];
    const float2 lA = h2f(((w << 4) & 0x00F000F0u) | 0x64006400u);  // bytes 0, 2
    const float2 lB = h2f(((w >> 4) & 0x00F000F0u) | 0x64006400u);  // bytes 1, 3
    const float2 hA = h2f((w & 0x00F000F0u) | 0x64006400u);
    const float2 hB = h2f(((w >> 8) & 0x00F000F0u) | 0x64006400u);
    const float2 l01 = fma2(make_float2(lA.x, lB.x), s0, c0), l23 = fma2(make_float2(lA.y, lB.y), s0, c0);
    const float2 h01 = fma2(make_float2(hA.x, hB.x), s1, c1), h23 = fma2(make_float2(hA.y, hB.y), s1, c1);
    o[2 * i] = pack_f16(l01.x, l01.y);
    o[2 * i + 1] = pack_f16(l23.x, l23.y);
    o[16 + 2 * i] = pack_f16(h01.x, h01.y);
    o[16 + 2 * i + 1] = pack_f16(h23.x, h23.y);
  }
}

// Four int8 times d, rounded once to f16: bytes biased to 1024 + (q + 128), the bias taken off
// exactly, then an f16 product (d is an f16, q an integer: the exact product is rounded once).
__device__ __forceinline__ void q80_word(uint32_t w, __half2 d, uint32_t& lo, uint32_t& hi) {
  const uint32_t x = w ^ 0x80808080u;
  const uint32_t a = __byte_perm(x, 0x64646464u, 0x4140), b = __byte_perm(x, 0x64646464u, 0x4342);
  const __half2 bias = __floats2half2_rn(1152.f, 1152.f);
  const __half2 r0 = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&a), bias), d);
  const __half2 r1 = __hmul2(__hsub2(*reinterpret_cast<const __half2*>(&b), bias), d);
  lo = *reinterpret_cast<const uint32_t*>(&r0);
  hi = *reinterpret_cast<const uint32_t*>(&r1);
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

template <int NT, int FMT>
__global__ void __launch_bounds__(kQmThreads, 1) kq_mma_kernel(const __grid_constant__ QmParams p) {
  using Cfg = QmCfg<NT, FMT>;
  constexpr int kPkStages = Cfg::kPkStages, kPkBytes = Cfg::kPkBytes, kUnit = Cfg::kUnit;
  constexpr int kAStages = Cfg::kAStages, kBStages = Cfg::kBStages, kBBytes = Cfg::kBBytes;
  constexpr int kBPer = Cfg::kBPer, kA0 = Cfg::kA0, kAccBufs = Cfg::kAccBufs;
  // a box dimension holds at most 256 elements: the 272-byte Q8_0 unit is mapped as 68 words
  constexpr int kBoxX = FMT == 12 ? 144 : 68;
  constexpr int kPkWarp = kQmExpWarps, kActWarp = kQmExpWarps + 1, kMmaWarp = kQmExpWarps + 2;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);

  uint64_t* pk_full = reinterpret_cast<uint64_t*>(smem);  // [kPkStages] two boxes landed
  uint64_t* pk_free = pk_full + kPkStages;                // [kPkStages] every expander warp left it
  uint64_t* a_full = pk_free + kPkStages;    // [kAStages] stored by the step's 8 warps
  uint64_t* a_free = a_full + kAStages;      // [kAStages] the MMAs that read it have retired
  uint64_t* b_full = a_free + kAStages;      // [kBStages] activations landed
  uint64_t* b_free = b_full + kBStages;      // [kBStages]
  uint64_t* acc_full = b_free + kBStages;    // [kAccBufs] a tile's products are complete
  uint64_t* acc_free = acc_full + kAccBufs;  // [kAccBufs] the epilogue has read them
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + kAccBufs);
  uint8_t* pk = smem + 1024;
  uint8_t* bstg = pk + kPkStages * kPkBytes;

  if (tid == 0) {
    for (int i = 0; i < kPkStages; ++i) {
      mbar_init(&pk_full[i], 1);
      mbar_init(&pk_free[i], kQmExpWarps);
    }
    for (int i = 0; i < kAStages; ++i) {
      mbar_init(&a_full[i], kQmExpWarps / 2);
      mbar_init(&a_free[i], 1);
    }
    for (int i = 0; i < kBStages; ++i) {
      mbar_init(&b_full[i], 1);
      mbar_init(&b_free[i], 1);
    }
    for (int i = 0; i < kAccBufs; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_free[i], kQmExpWarps);
    }
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
  const uint32_t tmem = *tmem_slot;
  const int njobs = qm_jobs(p.deal);
  bool ok = true;
  pdl_trigger();

  if (warp == kPkWarp) {
    // ================= weights: constant, so no wait on the previous kernel =====================
    if (tc_elect()) {
      const uint64_t pol = policy_evict_first();
      int n = 0;  // units brought so far
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
        for (int b = 0; b < job.n; ++b, ++n) {
          const int st = n % kPkStages;
          if (n >= kPkStages)
            ok = tc_wait(ok, &pk_free[st], (uint32_t)((n / kPkStages - 1) & 1), p.status);
          if (!ok) break;
          mbar_arrive_expect_tx(&pk_full[st], kPkBytes);
          uint8_t* dst = pk + (size_t)st * kPkBytes;
          tc_tma_box_2d(dst, tm0, (job.b0 + b) * kBoxX, y0, &pk_full[st], pol);
          tc_tma_box_2d(dst + kPkBytes / 2, tm1, (job.b0 + b) * kBoxX, y1, &pk_full[st], pol);
        }
      }
    }
    __syncwarp();
  } else if (warp == kActWarp) {
    // ================= activations: written by the kernel before this one =======================
    pdl_wait();
    if (tc_elect()) {
      int n = 0;
      for (int j = 0; j < njobs && ok; ++j) {
        const QmJob job = qm_job(p.deal, j);
        const uint8_t* src = p.xb + (size_t)job.b0 * 2 * kBPer * kBBytes;
        for (int s = 0; s < job.n * 2 * kBPer; ++s, ++n) {
          const int st = n % kBStages;
          if (n >= kBStages)
            ok = tc_wait(ok, &b_free[st], (uint32_t)((n / kBStages - 1) & 1), p.status);
          if (!ok) break;
          mbar_arrive_expect_tx(&b_full[st], kBBytes);
          bulk_g2s(bstg + (size_t)st * kBBytes, src + (size_t)s * kBBytes, kBBytes, &b_full[st]);
        }
      }
    }
    __syncwarp();
  } else if (warp == kMmaWarp) {
    // ================= MMA issue =================================================================
    if (tc_elect()) {
      int s = 0, h = 0;  // steps and activation stages so far
      for (int j = 0; j < njobs && ok; ++j) {
        const QmJob job = qm_job(p.deal, j);
        const int buf = j % kAccBufs;
        const uint32_t tmem_d = tmem + (uint32_t)(buf * NT);
        if (j >= kAccBufs) {
          ok = tc_wait(ok, &acc_free[buf], (uint32_t)((j / kAccBufs - 1) & 1), p.status);
          tc_after_sync();
        }
        for (int i = 0; i < 2 * job.n && ok; ++i, ++s) {
          const int st = s % kAStages;
          ok = tc_wait(ok, &a_full[st], (uint32_t)((s / kAStages) & 1), p.status);
          const uint32_t a_t = tmem + kA0 + (uint32_t)st * kQmACols;
#pragma unroll
          for (int hh = 0; hh < kBPer; ++hh, ++h) {
            const int bs = h % kBStages;
            ok = tc_wait(ok, &b_full[bs], (uint32_t)((h / kBStages) & 1), p.status);
            tc_after_sync();
            const uint32_t bbase = smem_u32(bstg + (size_t)bs * kBBytes);
            constexpr int kMma = kQmStepK / 16 / kBPer;  // K = 16 per instruction: 8 columns of A
#pragma unroll
            for (int m = 0; m < kMma; ++m)
              tc_mma_f16_ta(tmem_d, a_t + (hh * kMma + m) * 8,
                            tc_smem_desc(bbase + (m >> 2) * (NT * 128) + (m & 3) * 256, 128, 1024, 0),
                            p.idesc, (i > 0 || hh > 0 || m > 0) ? 1u : 0u);
            tc_commit(&b_free[bs]);
          }
          tc_commit(&a_free[st]);
        }
        tc_commit(&acc_full[buf]);
      }
    }
    __syncwarp();
  } else {
    // ================= dequantise into tensor memory, epilogue ==================================
    // lane quarter, 64-weight chunk of the step, which steps (0: even, 1: odd)
    const int q = warp & 3, c2 = (warp >> 2) & 1, grp = warp >> 3;
    const int c = 2 * grp + c2;  // chunk of the super-block: sub-blocks 2c, 2c+1
    // row of the tile that this tensor-memory lane holds: a gate/up tile has 16 gate rows and the
    // 16 up rows of the same outputs in every lane quarter
    const int erow = p.glu ? (lane & 15) + 16 * q + (lane >> 4) * 64 : q * 32 + lane;
    const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
    const uint32_t a_base = lane_base + kA0 + 32u * c2;

    // ---- epilogue of a job: this warp's NT / 4 tokens of its 32 lanes --------------------------
    auto epilogue = [&](int j) {
      const QmJob job = qm_job(p.deal, j);
      const int buf = j % kAccBufs;
      ok = tc_wait(ok, &acc_full[buf], (uint32_t)((j / kAccBufs) & 1), p.status);
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
#pragma unroll 1
      for (int g = 0; g < NT / 64; ++g) {  // 16 tokens at a time
        const int m0 = (warp >> 2) * (NT / 4) + 16 * g;
        if (m0 >= p.M) break;  // the same for the whole warp
        uint32_t v[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
              "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
              "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(lane_base + (uint32_t)(buf * NT + m0)));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        const int mc = min(16, p.M - m0);
        if (job.slot >= 0) {
          float* dst = p.part + (((size_t)blockIdx.x * 2 + job.slot) * NT + m0) * kQmRows + q * 32 + lane;
#pragma unroll
          for (int t = 0; t < 16; ++t)
            if (t < mc) dst[(size_t)t * kQmRows] = __uint_as_float(v[t]);
          continue;
        }
        float rs[16];
#pragma unroll
        for (int t = 0; t < 16; t += 4) {
          const float4 r4 = __ldcg(reinterpret_cast<const float4*>(p.rowscale + m0 + t));
          rs[t] = r4.x; rs[t + 1] = r4.y; rs[t + 2] = r4.z; rs[t + 3] = r4.w;
        }
        if (!p.glu) {
          const size_t o0 = (size_t)m0 * sg.ldy + row;
          if (row_ok) {
#pragma unroll
            for (int t = 0; t < 16; ++t)
              if (t < mc) {
                float r = __uint_as_float(v[t]) * rs[t];
                if (sg.residual) r = __fadd_rn(r, sg.residual[o0 + (size_t)t * sg.ldy]);
                sg.y[o0 + (size_t)t * sg.ldy] = r;
              }
          }
        } else {
          // gate lanes finish the even tokens, up lanes the odd ones
          const bool up = lane >= 16;
#pragma unroll
          for (int t = 0; t < 16; t += 2) {
            const float a = __uint_as_float(v[t]) * rs[t], b = __uint_as_float(v[t + 1]) * rs[t + 1];
            const float got = __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
            const float r = up ? glu_gate(got) * b : glu_gate(a) * got;
            const int tt = up ? t + 1 : t;
            if (row_ok && tt < mc) sg.y[(size_t)(m0 + tt) * sg.ldy + row] = r;
          }
        }
      }
      tc_before_sync();
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_free[buf]))
                     : "memory");
    };

    int n = 0;            // units so far
    int s = grp;          // this warp's steps: grp, grp + 2, ...
    int pending = -1;     // job whose epilogue is due
    bool waited = false;  // the epilogue reads what the previous kernel wrote (row scales, residual)
    for (int j = 0; j < njobs; ++j) {
      const int nu = qm_job(p.deal, j).n;
      for (int b = 0; b < nu; ++b, ++n, s += 2) {
        const int ps = n % kPkStages, st = s % kAStages;
        ok = tc_wait(ok, &pk_full[ps], (uint32_t)((n / kPkStages) & 1), p.status);
        uint32_t o[32];
        const uint8_t* blk = pk + (size_t)ps * kPkBytes + (size_t)erow * kUnit;
        if (FMT == 12) {
          // super-block of this row: f16 d, f16 dmin, 12 bytes of 6-bit scales and mins, 128 bytes
          // of nibbles (Hesper/Quantization/Q4_K_M.lean:13-52,120-144)
          const uint4 hdr = *reinterpret_cast<const uint4*>(blk);
          const uint4 qa = *reinterpret_cast<const uint4*>(blk + 16 + 32 * c);
          const uint4 qb = *reinterpret_cast<const uint4*>(blk + 32 + 32 * c);
          const float2 dd = h2f(hdr.x);
          // scale / min bytes j and j+1 (j = 2c) out of the 12 packed bytes hdr.y, hdr.z, hdr.w
          uint32_t sc2, m2;  // two 6-bit values each, in bytes 0 and 1
          const int sh = 16 * c2;
          if (grp == 0) {
            sc2 = (hdr.y >> sh) & 0x3F3Fu;
            m2 = (hdr.z >> sh) & 0x3F3Fu;
          } else {
            sc2 = ((hdr.w >> sh) & 0x0F0Fu) | ((hdr.y >> (sh + 2)) & 0x3030u);
            m2 = ((hdr.w >> (sh + 4)) & 0x0F0Fu) | ((hdr.z >> (sh + 2)) & 0x3030u);
          }
          const uint32_t qq[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
          q4k_expand(qq, dd.x * (float)(sc2 & 0xFF), dd.y * (float)(m2 & 0xFF),
                     dd.x * (float)(sc2 >> 8), dd.y * (float)(m2 >> 8), o);
        } else {
          // Q8_0 (Hesper/Layers/Linear.lean:6207-6223): blocks 2c and 2c+1 of the row's eight, 34
          // bytes each -- f16 d, then 32 int8.  The chunk starts on a word; block 2c's quants sit
          // two bytes into it (funnel shifts), block 2c+1's are word aligned.
          const uint32_t* wq = reinterpret_cast<const uint32_t*>(blk + 68 * c);
          uint32_t w[17];
#pragma unroll
          for (int i = 0; i < 17; ++i) w[i] = wq[i];
          const __half2 d0 = __half2half2(__ushort_as_half((unsigned short)(w[0] & 0xFFFFu)));
          const __half2 d1 = __half2half2(__ushort_as_half((unsigned short)(w[8] >> 16)));
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            q80_word(__funnelshift_r(w[i], w[i + 1], 16), d0, o[2 * i], o[2 * i + 1]);
            q80_word(w[9 + i], d1, o[16 + 2 * i], o[16 + 2 * i + 1]);
          }
        }
        if (s >= kAStages) {
          ok = tc_wait(ok, &a_free[st], (uint32_t)((s / kAStages - 1) & 1), p.status);
          tc_after_sync();
        }
        HB_TMEM_ST32(a_base + (uint32_t)st * kQmACols, o);
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&pk_free[ps]))
                       : "memory");
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_before_sync();
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&a_full[st]))
                       : "memory");
        // the A stages are refilled for this job: now the previous job's accumulator
        if (pending >= 0 && b == kAStages / 2 - 1) {
          if (!waited) pdl_wait();
          waited = true;
          epilogue(pending);
          pending = -1;
        }
      }
      if (pending >= 0) {
        if (!waited) pdl_wait();
        waited = true;
        epilogue(pending);
      }
      pending = j;
    }
    if (!waited) pdl_wait();
    if (pending >= 0) epilogue(pending);
  }
  tc_before_sync();
  __syncthreads();
  if (warp == kMmaWarp)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

// Adds the partials of the left-over tiles in K order and runs the epilogue on the sums.  One
// warp per (tile, token): 128 lanes' values as a float4 per lane.
__global__ void __launch_bounds__(256) kq_combine_kernel(const __grid_constant__ QmParams p, int NT,
                                                         int grid) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31, m = blockIdx.y * 8 + (threadIdx.x >> 5);
  const int t = blockIdx.x, nb = p.deal.nb, upc = p.deal.upc;
  const int c0 = t * nb / upc, c1 = ((t + 1) * nb - 1) / upc;
  if (m >= p.M || c0 == c1) return;  // one CTA did the whole tile and has stored it
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int cta = c0; cta <= c1; ++cta) {
    const int slot = t - cta * upc / nb;
    const float4 v = __ldcg(reinterpret_cast<const float4*>(
        p.part + (((size_t)cta * 2 + slot) * NT + m) * kQmRows + 4 * lane));
    a.x = __fadd_rn(a.x, v.x); a.y = __fadd_rn(a.y, v.y);
    a.z = __fadd_rn(a.z, v.z); a.w = __fadd_rn(a.w, v.w);
  }
  const float rs = __ldcg(p.rowscale + m);
  float r[4] = {a.x * rs, a.y * rs, a.z * rs, a.w * rs};
  const int tile = p.deal.W * grid + t;
  if (!p.glu) {
    int si = 0;
#pragma unroll
    for (int i = 1; i < kQmMaxSeg; ++i)
      if (i < p.nseg && tile >= p.seg[i].tile0) si = i;
    const QmSeg& sg = p.seg[si];
    const int row = (tile - sg.tile0) * kQmRows + 4 * lane;
    const size_t o = (size_t)m * sg.ldy + row;
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (row + e < sg.N) sg.y[o + e] = sg.residual ? __fadd_rn(r[e], sg.residual[o + e]) : r[e];
  } else {  // lanes 8q..8q+3 hold gate rows 16q.., lanes 8q+4..8q+7 their up rows
    const QmSeg& sg = p.seg[0];
    const int row = tile * 64 + 16 * (lane >> 3) + 4 * (lane & 3);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float up = __shfl_down_sync(0xffffffffu, r[e], 4);
      if (!(lane & 4) && row + e < sg.N) sg.y[(size_t)m * sg.ldy + row + e] = glu_gate(r[e]) * up;
    }
  }
}

}  // namespace hb

using namespace hb;

// Dealing `tiles` row tiles of `nb` super-blocks to the SMs: whole waves, then the rest cut into
// equal runs of units.  The rest stays whole (upc = nb) when cutting it saves less than the
// partials cost: a unit takes a CTA about max(800, 16 * (NT / 2 + 10)) cycles, partials and the
// second kernel about 3000 + 12 NT.
static QmDeal qm_deal(int tiles, int nb, int NT, int sms, int* grid) {
  QmDeal d = {tiles / sms, tiles % sms, nb, nb};
  if (d.R) {
    const int upc = (d.R * nb + sms - 1) / sms;
    const int unit = 16 * (NT / 2 + 10) > 800 ? 16 * (NT / 2 + 10) : 800;
    if ((long)(nb - upc) * unit > 3000 + 12 * NT) d.upc = upc;
  }
  *grid = d.W ? sms : (d.R * nb + d.upc - 1) / d.upc;
  return d;
}

template <int NT, int FMT>
static int kq_mma_launch(hb200_ctx* ctx, QmParams& p, int tiles, int nb, cudaStream_t st) {
  using Cfg = QmCfg<NT, FMT>;
  // kind::f16: D = f32, A and B f16, both K-major, N = NT, M = 128
  p.idesc = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(kQmRows >> 4) << 24);
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
  HB_CUDA(launch_pdl(kq_mma_kernel<NT, FMT>, dim3((unsigned)grid), dim3(kQmThreads),
                     (size_t)Cfg::kSmem, st, ctx->pdl, p));
  if (p.deal.R && p.deal.upc < nb)
    HB_CUDA(launch_pdl(kq_combine_kernel, dim3((unsigned)p.deal.R, (unsigned)((p.M + 7) / 8)), dim3(256),
                       0, st, ctx->pdl, p, NT, grid));
  return HB200_OK;
}

// For each of nseg tensors: y[m*ldy + n] = sum_k dequant(W)[n,k] x[m,k] (+ residual) for the
// M <= NT tokens staged by hb_gemm16_split (dtype f16, single term, NT token rows per block;
// NT = 64, 128 or 256), all in ONE product launch.  glu != 0: two tensors of equal shape, gate and
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
  p.xb = static_cast<const uint8_t*>(ctx->d_scratch) + kScratchLmSplit;
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
