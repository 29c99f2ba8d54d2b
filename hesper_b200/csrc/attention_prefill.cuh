// attention_prefill.cuh -- what the two prompt attention kernels share.
#pragma once

#include "common.cuh"

namespace hb {

constexpr int kPmRows = 64;  // query rows of a CTA of the mma.sync kernel

struct PmParams {
  const void* q;        // [nseq][T][H][D] f32 or f16
  const __half* k;      // [nseq][Hkv][slots][D]
  const __half* v;
  const int32_t* seqlens;  // [nseq] lengths after the T tokens
  float* out;           // [nseq][T][H][D], 8-byte aligned
  int q_is_f16;
  int nseq, T, H, Hkv, G, slots, window, ring;
  float scale_log2;
  // nsplit > 1: unnormalised partials and their (max, sum), for attn_prefill_merge_kernel
  int nsplit;
  float* part_o;   // [nseq][T][H][nsplit][D]
  float* part_ml;  // [nseq][T][H][nsplit][2]  (max in the exp2 domain, sum)
};

}  // namespace hb

// attention_prefill_mma.cu: the kernel without the merge
int hb_attn_prefill_mma(hb200_ctx* ctx, const hb::PmParams& p, int D, cudaStream_t st);
int hb_attn_prefill_mma_splits(const hb200_ctx* ctx, int nseq, int T, int G, int Hkv, int D, long span);
