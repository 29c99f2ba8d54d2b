// tcgen05.cuh -- small wrappers shared by the tensor-core kernels: shared-memory matrix
// descriptors, MMA issue / commit / fences, the 2-D tensor-map copy and the run-time lookup
// of the tensor-map encoder.
#pragma once

#include <cuda.h>  // CUtensorMap and its enums only; the encoder comes from the runtime

#include "common.cuh"

namespace hb {

// K-major shared-memory matrix descriptor.  layout 0: no swizzle, core matrices of 8 rows x
// 16 bytes, LBO = byte distance between core matrices adjacent in K, SBO = between 8-row
// groups.  layout 2: 128-byte swizzle, rows of 128 bytes in 1 KB atoms of 8 rows, SBO = 1024.
__device__ __forceinline__ uint64_t tc_smem_desc(uint32_t smem_addr, uint32_t lbo, uint32_t sbo,
                                                 uint32_t layout) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of this architecture
  d |= (uint64_t)layout << 61;
  return d;
}

// One lane of a converged warp, as a predicate ptxas can trace to elect.sync.  How an MMA loop is
// written decides what it costs (measured, M = 128, A in tensor memory, N = 64 / 128, cycles per
// MMA): behind `lane == 0` 132 whatever N; behind this predicate 42 / 74; with the whole warp
// converged and only the instruction itself predicated (tc_mma_f16_ta_w, tc_commit_w) 32 / 64, the
// tensor pipe's own rate -- descriptors are then computed in the uniform datapath.  A completed
// mbarrier costs 21 cycles through tc_wait_w and ~185 through the bounded loop of tc_wait.
__device__ __forceinline__ bool tc_elect() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\tselp.u32 %0, 1, 0, e;\n\t}"
      : "=r"(p));
  return p != 0;
}

__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tc_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

// kind::f16 with the A operand in tensor memory (lane = row, two 16-bit K elements per 32-bit
// column) and B through a shared-memory descriptor, and the commit, for a converged warp: every lane
// calls, one issues.  The MMA warp shares its
// scheduler with compute warps, so what an MMA costs is its instruction count: the descriptor's
// high word (no swizzle, LBO, SBO) and the instruction descriptor are immediates, and the low
// word -- smem address / 16 with LBO above it, tc_desc_lo -- is one addition per MMA.
__host__ __device__ constexpr uint32_t tc_desc_hi(uint32_t sbo) { return ((sbo >> 4) & 0x3FFF) | (1u << 14); }
__device__ __forceinline__ uint32_t tc_desc_lo(uint32_t smem_addr, uint32_t lbo) {
  return ((smem_addr & 0x3FFFF) >> 4) | ((lbo >> 4) << 16);
}
template <uint32_t kDescHi, uint32_t kIdesc>
__device__ __forceinline__ void tc_mma_f16_ta_w(uint32_t tmem_d, uint32_t tmem_a, uint32_t bdesc_lo,
                                                uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t.reg .b64 bd;\n\tmov.b64 bd, {%2, %3};\n\t"
      "elect.sync _|e, 0xffffffff;\n\tsetp.ne.b32 p, %5, 0;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], bd, %4, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "r"(bdesc_lo), "n"(kDescHi), "n"(kIdesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_commit_w(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(
          smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// One box of a 2-D tensor map into shared memory; completion is counted in bytes on `bar`.
// x in elements of the innermost dimension (x * element size must be a multiple of 16).
__device__ __forceinline__ void tc_tma_box_2d(void* dst, const CUtensorMap* tm, int x, int y,
                                              uint64_t* bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      ".L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(smem_u32(bar)), "l"(policy)
      : "memory");
}

// Bounded mbarrier wait for kernels whose whole life is microseconds: ~1e5 polls already
// means something is broken.  The kernel may be resident long before its predecessor ends (which may
// itself wait for another GPU), so a wait that depends on what the predecessor writes, directly or by
// way of another warp, only starts behind pdl_wait.  Once a wait has failed the later ones are skipped, so a broken
// launch ends quickly (and still releases its tensor memory).
__device__ __forceinline__ bool tc_wait(bool ok, uint64_t* bar, uint32_t parity, uint32_t* status) {
  if (!ok) return false;
#pragma unroll 1
  for (uint32_t it = 0; it < (1u << 17); ++it)
    if (mbar_try_wait(bar, parity)) return true;
  atomicOr(status, kStatusMbarTimeout);
  return false;
}

// The slow path of tc_wait_w: the barrier was not complete at the first look.
static __device__ __noinline__ bool tc_wait_slow(uint32_t bar, uint32_t parity, uint32_t* status) {
#pragma unroll 1
  for (uint32_t it = 0; it < (1u << 17); ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  atomicOr(status, kStatusMbarTimeout);
  return false;
}
// Bounded wait for the inner loops: one inline try, the loop out of line.  False when the bound
// ran out (the caller leaves its loop; what it would have produced never arrives, so the others'
// waits run out as well and the kernel ends).
__device__ __forceinline__ bool tc_wait_w(uint64_t* bar, uint32_t parity, uint32_t* status) {
  if (mbar_try_wait(bar, parity)) return true;
  return tc_wait_slow(smem_u32(bar), parity, status);
}

// Position in a ring of N stages and the parity of its current lap.  A consumer waits for parity
// `phase`; a producer waits for the stage to be free with parity `phase ^ 1`, which a fresh barrier
// passes at once.
template <int N>
struct TcRing {
  uint32_t i = 0, phase = 0;
  __device__ __forceinline__ void advance(int by = 1) {  // by <= N
    i += by;
    if (i >= N) {
      i -= N;
      phase ^= 1;
    }
  }
};

#define HB_TMEM_LD16(v, addr)                                                                  \
  asm volatile(                                                                                \
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "                                                \
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"                        \
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),    \
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),             \
        "=r"(v[13]), "=r"(v[14]), "=r"(v[15])                                                  \
      : "r"(addr))

#define HB_TMEM_LD32(v, addr)                                                                  \
  asm volatile(                                                                                \
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "                                                \
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"                                \
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"               \
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),    \
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),             \
        "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),          \
        "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),          \
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),          \
        "=r"(v[31])                                                                            \
      : "r"(addr))

#define HB_TMEM_ST32(addr, v)                                                                  \
  asm volatile(                                                                                \
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "                                          \
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"                               \
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(addr),         \
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),  \
      "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),        \
      "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]),      \
      "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]),      \
      "r"(v[29]), "r"(v[30]), "r"(v[31])                                                       \
      : "memory")

typedef CUresult (*TcEncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                    const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                    const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The tensor-map encoder is a driver entry point; it is looked up through the runtime so
// that the library does not link against the driver library.  Null when unavailable.
inline TcEncodeTiledFn tc_tensor_map_encoder() {
  static TcEncodeTiledFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<TcEncodeTiledFn>(f);
  }();
  return fn;
}

}  // namespace hb
