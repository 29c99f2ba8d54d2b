// bitlinear_mma.cu -- batched (16 tokens or more) ternary i2_s x int8 product on the 5th-generation
// tensor cores: tcgen05.mma kind::i8 with the int32 accumulator in tensor memory.
//
// Same arithmetic contract as the batch-1 kernel (bit-exact int32 accumulators, then
// y = ((float)acc*d)*s (+residual)); the reference's counterparts are the tiled and WMMA
// M>1 paths of BitLinear (Hesper/Layers/BitLinear.lean:122,869,994).  With 16 or more
// tokens per weight the op is a real contraction, so the weights are still streamed once
// but the multiply-accumulates move from dp4a to the tensor core:
//
//   quant_act_kernel   one CTA per token: optional RMSNorm, absmax int8 quantisation; the
//                      int8 activations are written straight in the shared-memory operand
//                      layout (K-major, 8x16-byte core matrices), one 8 KB block per
//                      128-wide K group, so the GEMM kernel fetches a B tile with ONE bulk copy
//   bitlinear_mma_kernel  one CTA per 128 weight rows, block of 64 or 128 tokens and K range, 20
//   warps with fixed roles (w = 0 the first behind the expanders):
//     * warp 3 copies the packed weights as boxes of 64 rows x 128 bytes (4 groups) through a 2-D
//       tensor map with the 128-byte swizzle, two per 16 KB slot of a 4-deep ring (per-row 1-D
//       bulk copies cost ~35 ns each at the TMA unit); warp 1 each step's activations with one bulk
//       copy.  Two warps: in one, a box was only asked for behind the waits of the activations;
//     * 16 warps in two groups that take the steps in turn expand two 128-wide groups per step
//       from 2-bit codes to unsigned bytes (0,1,2) and store them with tcgen05.st straight into
//       TENSOR MEMORY as the A operand (lane = weight row, 4 K-bytes per column): the expanded
//       weights never touch shared memory.  A step is a chain of ~1000 cycles of which its warps
//       issue a tenth: this chain, not the tensor pipe, is what a 64-token CTA waits for;
//     * warps 0 and 2 each issue the MMAs of every other step from one thread into their own
//       accumulator (tcgen05.mma kind::i8, A from tensor memory, B by a shared-memory
//       descriptor, M=128, N = tokens, K=32 per instruction).  One barrier per step gathers the 8
//       expander arrivals and the activation bytes; one tcgen05.commit per step releases the stage;
//     * epilogue: 16 warps read 32 lanes x 16 columns of both accumulators (tcgen05.ld 32x32b),
//       add them, subtract sum(q) per token (value = code - 1), scale and store.  A gate/up pair is
//       one launch: a tile holds 64 gate rows and the 64 up rows of the same outputs, a gate lane's
//       up value sits 16 lanes further in the same warp;
//     * split-K: each CTA publishes its int32 partial, the last to arrive (a ticket per tile and
//       token block) adds the others' and runs the epilogue -- exact, since integers commute.
// All tokens of a call (up to 512) go in one launch of each kernel: in passes of 128 a 256-token
// prompt paid both launches' latency twice.  Measured, 256 tokens, K=2560: q/k/v (3840 rows), o_proj,
// gate/up (2 x 6912, with the GLU) and down_proj (K=6912) together 150 -> 59 us.
// Every mbarrier wait is bounded; on expiry the kernel still releases its tensor memory.
#include "tcgen05.cuh"

namespace hb {

constexpr int kExpGroups = 2;   // groups of 8 expanding warps, taking the steps in turn
constexpr int kMmaThreads = kExpGroups * 256;
constexpr int kMmaRows = 128;    // weight rows per CTA = MMA M
constexpr int kChunkGroups = 4;  // 128-weight groups per packed box: 128 bytes of every row
constexpr int kPkStages = 4;     // packed ring
constexpr int kPkBytes = kMmaRows * kChunkGroups * 32;  // 16 KB box
constexpr int kStepGroups = 2;   // groups per pipeline step: one barrier round trip per 8 MMAs
constexpr int kAGroupCols = 32;  // TMEM columns of one expanded group: 128 K-bytes per row
constexpr int kMmaCtrl = 2048;   // barriers, tensor-memory slot, d[NT], sum(q)[NT]

// NT tokens of a CTA = MMA N: 64 or 128.  Tensor memory, 512 columns: accumulator of the first issuing warp at 0, the A stages
// behind it, the second warp's accumulator in the last NT columns.
template <int NT>
struct MmaCfg {
  static constexpr int kStages = NT == 64 ? 6 : 4;  // operand stages (A in TMEM, B in smem)
  static constexpr int kBBytes = NT * 128;          // activation tile of one 128-wide group
  static constexpr int kA0 = NT;                    // first column of the A stages
  static constexpr int kAcc1 = 512 - NT;            // the second accumulator
  static constexpr int kSmem = kMmaCtrl + kPkStages * kPkBytes + kStages * kStepGroups * kBBytes;
  // kind::i8: D = s32, A = u8, B = s8, both K-major, N = NT, M = 128
  static constexpr uint32_t kIdesc = (2u << 4) | (0u << 7) | (1u << 10) |
                                     ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(kMmaRows >> 4) << 24);
  static_assert(kA0 + kStages * kStepGroups * kAGroupCols <= kAcc1, "tensor memory columns");
  static_assert(kSmem <= 232448, "shared memory budget of one CTA");
};

struct MmaSeg {
  const uint8_t* w;
  const float* scale;
  const float* residual;
  float* y;
  int32_t* acc;
  int N;
  int tile0;
};

struct MmaParams {
  CUtensorMap tmap[4];  // per segment: packed weights as [N rows][K/4 bytes], boxes of 64 rows x 128
  MmaSeg seg[4];
  int nseg, K, M;
  int glu;             // seg 0 = gate, seg 1 = up: y = relu(gate)^2 * up into seg 0's y
  int ntb;             // blocks of NT tokens; CTA = (tile * nsplit + split) * ntb + token block
  int nsplit, gps;     // split-K: CTAs per tile, groups per split
  int32_t* part;       // [tile][token block][split][NT tokens][128 rows] partials (nsplit > 1)
  int* tickets;        // [tile][token block] arrival counters, zero between launches
  const uint8_t* xq;   // [token block][K/128][NT tokens x 128 bytes, core-matrix layout]
  const float* d;      // [ntb * NT] activation scales
  const int32_t* sumq; // [ntb * NT]
  uint32_t* status;
};

// ---- activation quantiser -------------------------------------------------------------

struct QuantParams {
  const float* x;      // [M][K]
  const float* gamma;  // nullable
  float eps;
  int K, M;
  uint8_t* xq;
  float* d;
  int32_t* sumq;
  float* act_scale;    // nullable user copy of d
  int bbytes;          // bytes of one 128-wide K group of a token block: NT x 128
};

__global__ void __launch_bounds__(256) quant_act_kernel(const __grid_constant__ QuantParams p) {
  __shared__ double red_d[8];
  __shared__ uint32_t red_u[8];
  __shared__ int red_i[8];
  extern __shared__ __align__(16) float xs[];  // [K]
  pdl_trigger();
  if (p.gamma)  // constants of the model: into L1 before the wait on the previous kernel
    for (int i = threadIdx.x * 32; i < p.K; i += 256 * 32)
      asm volatile("prefetch.global.L1 [%0];" ::"l"(p.gamma + i));
  pdl_wait();
  const int m = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int K = p.K, nvec = K >> 2;
  const int NT = p.bbytes >> 7, mt = m % NT;  // row of its token block
  uint8_t* const xq = p.xq + (size_t)(m / NT) * (K >> 7) * p.bbytes;
  auto dst_of = [&](int i) {  // float4 index -> byte offset of its 4 int8 in the operand layout
    const int k = i << 2;
    return (size_t)(k >> 7) * p.bbytes + (size_t)(mt >> 3) * 1024 + (size_t)((k & 127) >> 4) * 128 +
           (size_t)(mt & 7) * 16 + (k & 15);
  };
  if (m >= p.M) {  // padding token of the tile
    for (int i = tid; i < nvec; i += 256) *reinterpret_cast<uint32_t*>(xq + dst_of(i)) = 0u;
    if (tid == 0) {
      p.d[m] = 0.f;
      p.sumq[m] = 0;
    }
    return;
  }
  const float4* xg = reinterpret_cast<const float4*>(p.x + (size_t)m * K);
  float4* x4 = reinterpret_cast<float4*>(xs);
  float amax = 0.f;
  if (p.gamma) {
    double ss = 0.0;
    for (int i = tid; i < nvec; i += 256) {
      const float4 v = __ldcg(xg + i);
      x4[i] = v;
      ss += (double)v.x * v.x + (double)v.y * v.y + (double)v.z * v.z + (double)v.w * v.w;
    }
    ss = warp_sum(ss);
    if (lane == 0) red_d[warp] = ss;
    __syncthreads();
    ss = 0.0;
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += red_d[i];
    const float rinv = (float)(1.0 / sqrt(ss / (double)K + (double)p.eps));
    const float4* gg = reinterpret_cast<const float4*>(p.gamma);
    for (int i = tid; i < nvec; i += 256) {
      float4 v = x4[i];
      const float4 g = __ldg(gg + i);
      v.x = __fmul_rn(__fmul_rn(v.x, rinv), g.x);
      v.y = __fmul_rn(__fmul_rn(v.y, rinv), g.y);
      v.z = __fmul_rn(__fmul_rn(v.z, rinv), g.z);
      v.w = __fmul_rn(__fmul_rn(v.w, rinv), g.w);
      x4[i] = v;
      amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
    }
  } else {
    for (int i = tid; i < nvec; i += 256) {
      const float4 v = __ldcg(xg + i);
      x4[i] = v;
      amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
    }
  }
  const uint32_t wmax = __reduce_max_sync(0xffffffffu, __float_as_uint(amax));
  if (lane == 0) red_u[warp] = wmax;
  __syncthreads();
  uint32_t mx = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) mx = max(mx, red_u[i]);
  amax = __uint_as_float(mx);
  const float d = __fdiv_rn(amax, 127.0f);
  const float inv = amax == 0.f ? 0.f : __fdiv_rn(127.0f, amax);
  int sumq = 0;
  for (int i = tid; i < nvec; i += 256) {
    const float4 v = x4[i];
    const int q0 = __float2int_rn(__fmul_rn(v.x, inv)), q1 = __float2int_rn(__fmul_rn(v.y, inv));
    const int q2 = __float2int_rn(__fmul_rn(v.z, inv)), q3 = __float2int_rn(__fmul_rn(v.w, inv));
    sumq += (q0 + q1) + (q2 + q3);
    *reinterpret_cast<uint32_t*>(xq + dst_of(i)) =
        (uint32_t)(q0 & 0xff) | ((uint32_t)(q1 & 0xff) << 8) | ((uint32_t)(q2 & 0xff) << 16) |
        ((uint32_t)q3 << 24);
  }
  sumq = __reduce_add_sync(0xffffffffu, sumq);
  if (lane == 0) red_i[warp] = sumq;
  __syncthreads();
  if (tid == 0) {
    int s = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += red_i[i];
    p.d[m] = d;
    p.sumq[m] = s;
    if (p.act_scale) p.act_scale[m] = d;
  }
}

// ---- tcgen05 helpers --------------------------------------------------------------------

// A operand from tensor memory (lane = weight row, 4 K-bytes per 32-bit column).
__device__ __forceinline__ void umma_i8_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc,
                                           uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

template <int NT>
__global__ void __launch_bounds__(kMmaThreads + 128, 1)
    bitlinear_mma_kernel(const __grid_constant__ MmaParams p) {
  using Cfg = MmaCfg<NT>;
  constexpr int kStages = Cfg::kStages, kBBytes = Cfg::kBBytes;
  constexpr int NCH = NT / 64;  // 16-token chunks an epilogue warp owns
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // this CTA's K range (split-K over 128-wide groups; a whole row when nsplit == 1)
  const int tb = (int)blockIdx.x % p.ntb, ts = (int)blockIdx.x / p.ntb;
  const int tile = ts / p.nsplit, split = ts % p.nsplit;
  const int M = min(NT, p.M - tb * NT);  // tokens of this block
  const uint8_t* const xq = p.xq + (size_t)tb * (p.K >> 7) * Cfg::kBBytes;
  const int gbase = split * p.gps;
  const int ngroups = min(p.gps, (p.K >> 7) - gbase);
  const int nchunks = (ngroups + kChunkGroups - 1) / kChunkGroups;
  const int nsteps = (ngroups + kStepGroups - 1) / kStepGroups;
  constexpr int kExpWarps = kMmaThreads / 32;  // these expand; then MMA, copy, MMA, copy
  constexpr int kMmaWarp = kExpWarps, kActWarp = kExpWarps + 1, kPkWarp = kExpWarps + 3;

  // control block, then the packed ring and the activation stages (1 KB aligned)
  uint64_t* pk_full = reinterpret_cast<uint64_t*>(smem);  // [kPkStages] box landed (tx bytes)
  uint64_t* pk_free = pk_full + kPkStages;                 // [kPkStages] every expander warp left it
  uint64_t* full = pk_free + kPkStages;   // [kStages] A stored by a group's 8 warps + B landed (tx bytes)
  uint64_t* mma_done = full + kStages;    // [kStages] the MMAs that read the stage have retired
  uint64_t* done = mma_done + kStages;    // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  float* sd = reinterpret_cast<float*>(smem + 512);        // [NT]
  int* ssum = reinterpret_cast<int*>(smem + 1024);         // [NT]
  uint8_t* pk = smem + kMmaCtrl;
  uint8_t* bstg = pk + kPkStages * kPkBytes;  // [kStages][kStepGroups] activation tiles

  // tile -> (segment, first row)
  int seg = 0;
  if (!p.glu) {
#pragma unroll
    for (int s = 1; s < 4; ++s)
      if (s < p.nseg && tile >= p.seg[s].tile0) seg = s;
  }
  const int seg_N = p.seg[seg].N;
  // a gate/up tile holds 64 gate rows and the 64 up rows of the same outputs
  const int row0 = p.glu ? tile * 64 : (tile - p.seg[seg].tile0) * kMmaRows;

  if (tid == 0) {
    for (int i = 0; i < kPkStages; ++i) {
      mbar_init(&pk_full[i], 1);
      mbar_init(&pk_free[i], kExpWarps);  // a box is two steps: one of each group
    }
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&full[i], 8 + 1);
      mbar_init(&mma_done[i], 1);
    }
    mbar_init(done, 2);
    fence_mbar_init();
  }
  if (warp == kMmaWarp) {  // all 512 columns: two accumulators, the A stages between them
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
        smem_u32(tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_before_sync();
  __syncthreads();
  tc_after_sync();
  const uint32_t tmem = *tmem_slot;
  bool ok = true;
  pdl_trigger();

  if (warp == kPkWarp) {
    // ================= packed weight boxes: constant, so no wait on the previous kernel ==========
    // A warp of its own: behind the activations' waits a box was only asked for when it was needed
    // (K=6912 unsplit, 64 tokens: 37 us).
    const uint64_t pol = policy_evict_first();
    const CUtensorMap* tm = &p.tmap[seg];
    const CUtensorMap* tm1 = p.glu ? &p.tmap[1] : tm;
    const int row1 = p.glu ? row0 : row0 + 64;
    TcRing<kPkStages> r;
    for (int c = 0; c < nchunks; ++c, r.advance()) {
      // a slot is freed by way of a product once the A stages are full: bounded waits, see tc_wait
      if (c == kPkStages + kStages / kExpGroups) pdl_wait();
      ok = tc_wait_w(&pk_free[r.i], r.phase ^ 1, p.status);
      if (!ok) break;
      if (tc_elect()) {  // two halves of 64 rows
        uint8_t* dst = pk + (size_t)r.i * kPkBytes;
        const int x = (gbase + c * kChunkGroups) * 32;
        mbar_arrive_expect_tx(&pk_full[r.i], kPkBytes);
        tc_tma_box_2d(dst, tm, x, row0, &pk_full[r.i], pol);
        tc_tma_box_2d(dst + kPkBytes / 2, tm1, x, row1, &pk_full[r.i], pol);
      }
      __syncwarp();
    }
  } else if (warp == kActWarp) {
    // ================= activation tiles: written by the kernel before this one ===================
    pdl_wait();
    TcRing<kStages> r;
    for (int s = 0; s < nsteps; ++s, r.advance()) {
      ok = tc_wait_w(&mma_done[r.i], r.phase ^ 1, p.status);  // the MMAs that read the stage last
      if (!ok) break;
      if (tc_elect()) {  // the step's groups are contiguous in the operand layout
        const int g0 = s * kStepGroups;
        const uint32_t bytes = (uint32_t)min(kStepGroups, ngroups - g0) * kBBytes;
        mbar_arrive_expect_tx(&full[r.i], bytes);
        bulk_g2s(bstg + (size_t)r.i * kStepGroups * kBBytes, xq + (size_t)(gbase + g0) * kBBytes, bytes,
                 &full[r.i]);
      }
      __syncwarp();
    }
  } else if (warp == kMmaWarp || warp == kMmaWarp + 2) {
    // ================= two MMA warps: even steps -> accumulator 0, odd steps -> accumulator 1
    const int which = warp == kMmaWarp ? 0 : 1;
    const uint32_t tmem_d = tmem + (which ? (uint32_t)Cfg::kAcc1 : 0u);
    pdl_wait();  // the activations come behind it: the waits below are bounded by this kernel's own work
    if (tc_elect()) {
      for (int s = which; s < nsteps; s += 2) {
        const int st = s % kStages;
        ok = ok && tc_wait_w(&full[st], (uint32_t)((s / kStages) & 1), p.status);
        tc_after_sync();
        const uint32_t a_t = tmem + Cfg::kA0 + (uint32_t)st * (kStepGroups * kAGroupCols);
        const uint32_t bbase = smem_u32(bstg + (size_t)st * kStepGroups * kBBytes);
        const int ng = min(kStepGroups, ngroups - s * kStepGroups);
#pragma unroll
        for (int gg = 0; gg < kStepGroups; ++gg)
          if (gg < ng) {
#pragma unroll
            for (int j = 0; j < 4; ++j)  // K = 32 bytes per instruction: 8 columns of A
              umma_i8_ta(tmem_d, a_t + gg * kAGroupCols + j * 8,
                         tc_smem_desc(bbase + gg * kBBytes + j * 256, 128, 1024, 0), Cfg::kIdesc,
                         (s > 1 || gg > 0 || j > 0) ? 1u : 0u);
          }
        tc_commit(&mma_done[st]);  // arrives once these (and all earlier) MMAs have retired
      }
      tc_commit(done);
    }
    __syncwarp();
  } else {
    // ================= expander warps ========================================================
    // warp w of a group owns TMEM lanes (= weight rows) 32*(w&3).., and K-half h = w>>2 of every
    // 128-wide group: planes 2h and 2h+1 of the packed bytes = K bytes 64h..64h+63 = 16 columns.
    static_assert(kExpGroups * kStepGroups == kChunkGroups, "a box is one step of every group");
    const int q = warp & 3, h = (warp >> 2) & 1, grp = warp >> 3;
    // row of the box that this lane expands: a gate/up tile has 16 gate rows and the 16 up rows
    // of the same outputs in every lane quarter
    const int erow = p.glu ? (lane & 15) + 16 * q + (lane >> 4) * 64 : q * 32 + lane;
    const uint32_t lane_addr = tmem + ((uint32_t)(q * 32) << 16) + Cfg::kA0 + 16u * h;
    for (int s = grp; s < nsteps; s += kExpGroups) {
      const int st = s % kStages, c = s / kExpGroups;
      if (s >= kStages) {
        if (s < kStages + kExpGroups) pdl_wait();  // freed by a product, which needs the activations
        ok = ok && tc_wait_w(&mma_done[st], (uint32_t)(((s / kStages) - 1) & 1), p.status);
        tc_after_sync();
      }
      ok = ok && tc_wait_w(&pk_full[c % kPkStages], (uint32_t)((c / kPkStages) & 1), p.status);
      const int ng = min(kStepGroups, ngroups - s * kStepGroups);
#pragma unroll
      for (int gg = 0; gg < kStepGroups; ++gg) {
        if (gg >= ng) break;
        const int gi = grp * kStepGroups + gg;  // group of the box
        // the row's 32 packed bytes of this group: units 2gi and 2gi+1 of its swizzled 128 bytes
        const uint8_t* rowp = pk + (size_t)(c % kPkStages) * kPkBytes + (size_t)erow * 128;
        const uint4 w0 = *reinterpret_cast<const uint4*>(rowp + (((2 * gi) ^ (erow & 7)) << 4));
        const uint4 w1 = *reinterpret_cast<const uint4*>(rowp + (((2 * gi + 1) ^ (erow & 7)) << 4));
        const uint32_t w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
        uint32_t o[16];
#pragma unroll
        for (int pp = 0; pp < 2; ++pp) {
          // plane pl holds elements 32*pl + j in byte j: word i -> K bytes 32*pl + 4i .. +3
          const int sh = h ? (2 - 2 * pp) : (6 - 2 * pp);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[8 * pp + i] = (w[i] >> sh) & 0x03030303u;
        }
        const uint32_t taddr = lane_addr + (uint32_t)st * (kStepGroups * kAGroupCols) +
                               (uint32_t)gg * kAGroupCols;
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
            "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
            "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]),
            "r"(o[8]), "r"(o[9]), "r"(o[10]), "r"(o[11]), "r"(o[12]), "r"(o[13]), "r"(o[14]),
            "r"(o[15])
            : "memory");
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&pk_free[c % kPkStages]);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[st]);
    }
    pdl_wait();  // d and sum(q) come from the quantiser
    if (tid < NT) {
      sd[tid] = p.d[tb * NT + tid];
      ssum[tid] = p.sumq[tb * NT + tid];
    }
  }
  pdl_wait();
  ok = tc_wait(true, done, 0, p.status) && ok;
  tc_after_sync();
  __syncthreads();  // sd / ssum visible; every warp past its loop

  // ---- epilogue: TMEM lane = weight row, column = token.  Warps w, w + 4, w + 8, w + 12 share a
  //      lane quarter; a warp owns the 16-token chunks (w >> 2), (w >> 2) + 4, ... -------------
  const int q = warp & 3, half = warp >> 2;  // lane quarter, first chunk (expander warps only)
  const int r = q * 32 + lane;
  uint32_t v[NCH][16];
  if (warp < kExpWarps) {
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)((half + 4 * c) * 16);
      HB_TMEM_LD16(v[c], taddr);
      if (nsteps > 1) {  // the second MMA warp's accumulator
        uint32_t u[16];
        HB_TMEM_LD16(u, taddr + (uint32_t)Cfg::kAcc1);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int t = 0; t < 16; ++t) v[c][t] += u[t];
      } else {
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      }
    }
  }

  // ---- split-K: publish the int32 partial, the last split of the tile to arrive adds them ---
  // Integer addition commutes, so the result is bit-identical to the unsplit product.
  bool finish = true;
  if (p.nsplit > 1) {
    __shared__ int s_last;
    const int tk = tile * p.ntb + tb;
    int32_t* mine = p.part + ((size_t)(tk * p.nsplit + split) * NT) * kMmaRows;
    if (warp < kExpWarps) {
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        const int m0 = (half + 4 * c) * 16;
        if (m0 >= M) continue;
#pragma unroll
        for (int t = 0; t < 16; ++t) mine[(size_t)(m0 + t) * kMmaRows + r] = (int32_t)v[c][t];
      }
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      const int t = atomicAdd(&p.tickets[tk], 1);
      s_last = (t == p.nsplit - 1);
      if (s_last) p.tickets[tk] = 0;  // every split has arrived: ready for the next launch
    }
    __syncthreads();
    finish = s_last != 0;
    if (finish && warp < kExpWarps) {
      __threadfence();
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        const int m0 = (half + 4 * c) * 16;
        if (m0 >= M) continue;
        for (int s2 = 0; s2 < p.nsplit; ++s2) {
          if (s2 == split) continue;
          const int32_t* other = p.part + ((size_t)(tk * p.nsplit + s2) * NT + m0) * kMmaRows + r;
#pragma unroll
          for (int t = 0; t < 16; ++t) v[c][t] += (uint32_t)__ldcg(other + (size_t)t * kMmaRows);
        }
      }
    }
  }

  if (finish && warp < kExpWarps) {
    const bool up = p.glu && lane >= 16;
    const int row = p.glu ? row0 + 16 * q + (lane & 15) : row0 + r;
    const bool row_ok = ok && row < seg_N;
    const float ws = __ldg(p.seg[up ? 1 : seg].scale);
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const int m0 = (half + 4 * c) * 16;
      if (m0 >= M) continue;  // the same for the whole warp
      const int mcount = min(16, M - m0);
      const size_t o0 = (size_t)(tb * NT + m0) * seg_N + row;
      float* yp = p.seg[seg].y + o0;
      const float* rp = p.seg[seg].residual ? p.seg[seg].residual + o0 : nullptr;
      int32_t* ap = p.seg[seg].acc ? p.seg[seg].acc + o0 : nullptr;
      // all shared-memory reads first (v[t] becomes the integer total), so that the stores
      // below, whose target the compiler cannot tell from shared memory, do not serialise them
      float dsc[16];
#pragma unroll
      for (int t = 0; t < 16; ++t) {
        v[c][t] = (uint32_t)((int)v[c][t] - ssum[m0 + t]);
        dsc[t] = sd[m0 + t];
      }
      if (p.glu) {
        // gate lanes finish the even tokens, up lanes (16 further) the odd ones
#pragma unroll
        for (int t = 0; t < 16; t += 2) {
          const float a = __fmul_rn(__fmul_rn((float)(int)v[c][t], dsc[t]), ws);
          const float b = __fmul_rn(__fmul_rn((float)(int)v[c][t + 1], dsc[t + 1]), ws);
          const float got = __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
          const float gt = up ? got : a, rl = gt > 0.f ? gt : 0.f;
          const float y = __fmul_rn(__fmul_rn(rl, rl), up ? b : got);
          const int tt = up ? t + 1 : t;
          if (row_ok && tt < mcount) yp[(size_t)tt * seg_N] = y;
        }
        continue;
      }
      if (!row_ok) continue;
      if (ap) {
#pragma unroll
        for (int t = 0; t < 16; ++t)
          if (t < mcount) ap[(size_t)t * seg_N] = (int)v[c][t];
      }
      float res[16];
      if (rp) {
#pragma unroll
        for (int t = 0; t < 16; ++t) res[t] = t < mcount ? rp[(size_t)t * seg_N] : 0.f;
      }
#pragma unroll
      for (int t = 0; t < 16; ++t)
        if (t < mcount) {
          float y = __fmul_rn(__fmul_rn((float)(int)v[c][t], dsc[t]), ws);
          if (rp) y = __fadd_rn(y, res[t]);
          yp[(size_t)t * seg_N] = y;
        }
    }
  }
  tc_before_sync();
  __syncthreads();
  if (warp == kMmaWarp)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

}  // namespace hb

using namespace hb;

// How a launch is dealt: token blocks of NT, K ranges per tile.  A block of 64 tokens more costs
// only its own CTA (the weights come from L2), so it is preferred until the CTAs need a second
// wave; cutting K pays for few tiles with a long K alone, partials and their fence cost 2 to 4
// us.  Measured (us, quantiser included; block/K ranges): K=2560 N=2560 at 128 tokens 64/1 9.0, 64/2
// 10.5, 128/1 10.8, 128/5 15.5; K=6912 N=2560 at 128 tokens 64/1 16.7, 64/3 15.0, 128/2 17.8, at 256
// 64/1 19.4, 128/2 22.3; K=2560 N=6912 gate/up at 128 tokens 64/1 (216 CTAs) 16.1, 128/1 11.0.  The
// cost below is in cycles, fitted to these.
struct BlDeal {
  int NT, ntb, nsplit, gps;
};
static BlDeal bl_deal(const hb200_ctx* ctx, int tiles, int ngroups, int M) {
  BlDeal best = {};
  long best_cost = 0;
  for (int NT = 64; NT <= (M > 64 ? 128 : 64); NT *= 2) {
    const int ntb = (M + NT - 1) / NT;
    for (int ns = 1; ns <= (ngroups >= 8 ? ngroups / 4 : 1); ++ns) {  // at least two steps each
      const long ctas = (long)tiles * ntb * ns;
      if (ns > 1 && (ctas > ctx->sm_count || tiles * ntb > kCtxTickets ||
                     (size_t)ctas * NT * kMmaRows * 4 > kScratchBytes - kScratchSplitK))
        break;
      const int gps = (ngroups + ns - 1) / ns;
      const long waves = (ctas + ctx->sm_count - 1) / ctx->sm_count;
      const long cost = waves * (4500 + 220L * gps + (NT == 128 ? 3500 : 0)) +
                        (ns > 1 ? 4500 + 11L * ns * NT : 0);
      if (best.NT == 0 || cost < best_cost) {
        best_cost = cost;
        best = {NT, ntb, (ngroups + gps - 1) / gps, gps};  // no empty split
      }
    }
  }
  return best;
}

template <int NT>
static int bl_mma_launch(hb200_ctx* ctx, MmaParams& p, int tiles, cudaStream_t st) {
  const int rc = hb_func_smem(ctx, reinterpret_cast<const void*>(bitlinear_mma_kernel<NT>),
                              (size_t)MmaCfg<NT>::kSmem);
  if (rc != HB200_OK) return rc;
  HB_CUDA(launch_pdl(bitlinear_mma_kernel<NT>, dim3(tiles * p.nsplit * p.ntb), dim3(kMmaThreads + 128),
                     (size_t)MmaCfg<NT>::kSmem, st, ctx->pdl, p));
  return HB200_OK;
}

// Batched path of the ternary products: 1 <= M <= kBlMmaTokens tokens in one launch of the
// quantiser and one of the product.  glu: two tensors of equal shape, gate and up, and segs[0].d_y
// = relu(gate)^2 * up.  Scratch in the context: quantised activations in operand layout, their
// scales and sums, split-K partials.
int hb_bitlinear_mma_run(hb200_ctx* ctx, const hb200_bitlinear_seg* segs, int nseg, int K, int glu,
                         const float* d_x, int M, const float* d_rms_gamma, float rms_eps,
                         float* d_act_scale, cudaStream_t st) {
  ScratchUse use(ctx, st);  // quantised activation tiles, split-K partials, tickets
  HB_REQUIRE(M >= 1 && M <= kBlMmaTokens, "bitlinear (batched): %d tokens in one pass (at most %d)", M,
             kBlMmaTokens);
  HB_REQUIRE(!glu || (nseg == 2 && segs[0].N == segs[1].N), "bitlinear (batched): gate and up differ in shape");
  MmaParams p = {};
  int t = 0;
  TcEncodeTiledFn encode = tc_tensor_map_encoder();
  HB_REQUIRE(encode != nullptr, "bitlinear (batched): the driver has no cuTensorMapEncodeTiled");
  for (int s = 0; s < nseg; ++s) {
    p.seg[s] = {static_cast<const uint8_t*>(segs[s].d_packed), segs[s].d_scale,
                segs[s].d_residual, segs[s].d_y, segs[s].d_acc, segs[s].N, t};
    t += (segs[s].N + kMmaRows - 1) / kMmaRows;
    HB_REQUIRE((reinterpret_cast<uintptr_t>(segs[s].d_packed) & 15) == 0,
               "bitlinear (batched): packed weights must be 16-byte aligned");
    const cuuint64_t dims[2] = {(cuuint64_t)(K / 4), (cuuint64_t)segs[s].N};
    const cuuint64_t strides[1] = {(cuuint64_t)(K / 4)};  // bytes between rows
    const cuuint32_t box[2] = {(cuuint32_t)(kChunkGroups * 32), (cuuint32_t)(kMmaRows / 2)};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult rc = encode(&p.tmap[s], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2,
                               const_cast<void*>(segs[s].d_packed), dims, strides, box, estr,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    HB_REQUIRE(rc == CUDA_SUCCESS, "bitlinear (batched): cuTensorMapEncodeTiled failed (%d)",
               (int)rc);
  }
  if (glu) t = (segs[0].N + kMmaRows / 2 - 1) / (kMmaRows / 2);
  const BlDeal deal = bl_deal(ctx, t, K / 128, M);
  const int slots = deal.ntb * deal.NT;  // token slots, padding included
  HB_REQUIRE(4096 + (size_t)slots * K <= kScratchLmSplit,
             "bitlinear (batched): K=%d needs %zu bytes of activation scratch", K, (size_t)slots * K);
  uint8_t* base = static_cast<uint8_t*>(ctx->d_scratch);
  float* d = reinterpret_cast<float*>(base);                // [kBlMmaTokens]
  int32_t* sumq = reinterpret_cast<int32_t*>(base + 2048);  // [kBlMmaTokens]
  uint8_t* xq = base + 4096;
  QuantParams q = {d_x, d_rms_gamma, rms_eps, K, M, xq, d, sumq, d_act_scale, deal.NT * 128};
  HB_CUDA(launch_pdl(quant_act_kernel, dim3(slots), dim3(256), (size_t)K * sizeof(float), st,
                     ctx->pdl, q));
  p.nseg = nseg;
  p.K = K;
  p.M = M;
  p.glu = glu;
  p.ntb = deal.ntb;
  p.nsplit = deal.nsplit;
  p.gps = deal.gps;
  p.part = reinterpret_cast<int32_t*>(base + kScratchSplitK);
  p.tickets = ctx->d_tickets;
  p.xq = xq;
  p.d = d;
  p.sumq = sumq;
  p.status = ctx->d_status;
  return deal.NT == 64 ? bl_mma_launch<64>(ctx, p, t, st) : bl_mma_launch<128>(ctx, p, t, st);
}
