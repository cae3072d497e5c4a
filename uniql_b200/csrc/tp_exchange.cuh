// Cross-GPU steps of a decode launch's epilogue (see CommView): four adjacent columns of one batch row at a time, always
// as epoch-tagged 8-byte words stored into the consumer's memory.  Shared by the two kernels that run decode launches, so
// that the words of a launch are the same whichever of them a rank runs.
#pragma once

#include "linear_internal.cuh"

namespace uniql {

constexpr int kTpSpinLimit = 1 << 22;     // polls of a word another GPU has to write before giving up

__device__ __forceinline__ void tp_st_word(uint2* p, uint32_t data, uint32_t flag) {
  asm volatile("st.relaxed.sys.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(data), "r"(flag) : "memory");
}
__device__ __forceinline__ uint4 tp_ld_word2(const uint2* p) {   // two adjacent {data, epoch} words
  uint4 v;
  asm volatile("ld.relaxed.sys.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}

// Epoch counters live on the device (CUDA-graph replay safe): one per 64-column block for the sum, one per rank for the
// feature area.  The words of a launch carry counter + 1; the launch advances a block's counter when it has finished the
// block, the consumer of the gathered row advances the other.
__device__ __forceinline__ volatile uint32_t* tp_reduce_counter(const CommView& cv, int block) {
  return reinterpret_cast<volatile uint32_t*>(cv.bufs[cv.rank] + cv.reduce_epoch_off + 4 * (size_t)block);
}
__device__ __forceinline__ uint32_t tp_gather_epoch(const CommView& cv) {
  return *reinterpret_cast<const volatile uint32_t*>(cv.bufs[cv.rank] + cv.gather_epoch_off) + 1;
}

// Row-parallel shard: where a rank would store its fp16 result it stores the partial into every rank's staging block
// (addressed per 64-column block: 16 rows x 32 words; c: column inside the block) ...
__device__ __forceinline__ void tp_push4(const CommView& cv, uint32_t ep, int block, int m, int c, float4 v) {
  const __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
  const size_t word = (size_t)block * kFuseBlockWords + (size_t)m * 32 + (c >> 1);
  const size_t slot = ((size_t)(ep & 1u) * cv.world + cv.rank) * (size_t)cv.block_cap * kFuseBlockWords + word;
  for (int r = 0; r < cv.world; ++r) {
    uint2* dst = reinterpret_cast<uint2*>(cv.bufs[r] + cv.reduce_off) + slot;
    tp_st_word(dst, *reinterpret_cast<const uint32_t*>(&lo), ep);
    tp_st_word(dst + 1, *reinterpret_cast<const uint32_t*>(&hi), ep);
  }
}
// ... and then adds up the words of all ranks that arrived in its own block (bounded wait, rank order, fp32: the same
// bits on every rank).  The first look at AHEAD ranks' words goes out together (one round trip instead of one per rank; a
// look holds four registers); a word that has not arrived yet is then polled on its own.
template <int AHEAD>
__device__ __forceinline__ float4 tp_gather4(const CommView& cv, uint32_t ep, int block, int m, int c, bool& failed) {
  float4 acc4 = make_float4(0.f, 0.f, 0.f, 0.f);
  const size_t word = (size_t)block * kFuseBlockWords + (size_t)m * 32 + (c >> 1);
  const size_t rstride = (size_t)cv.block_cap * kFuseBlockWords;
  const uint2* base = reinterpret_cast<const uint2*>(cv.bufs[cv.rank] + cv.reduce_off) +
                      (size_t)(ep & 1u) * cv.world * rstride + word;
#pragma unroll 1
  for (int r0 = 0; r0 < cv.world; r0 += AHEAD) {
    uint4 w[AHEAD];
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
      if (r0 + i < cv.world) w[i] = tp_ld_word2(base + (size_t)(r0 + i) * rstride);
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
      if (r0 + i < cv.world) {
        int spin = 0;
        while ((w[i].y != ep || w[i].w != ep) && !failed) {
          if (++spin > kTpSpinLimit) { failed = true; break; }
          w[i] = tp_ld_word2(base + (size_t)(r0 + i) * rstride);
        }
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&w[i].x));
        const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&w[i].z));
        acc4.x += a.x; acc4.y += a.y; acc4.z += b.x; acc4.w += b.y;
      }
  }
  return acc4;
}

// Column shard: the finished columns n..n + 3 also go into every rank's feature area (only real columns travel; n_out is
// even).
__device__ __forceinline__ void tp_feature4(const CommView& cv, uint32_t ep, int m, int n, int n_out, const __half (&h)[4]) {
  const size_t word = ((size_t)(ep & 1u) * 16 + m) * (size_t)(cv.feat_cap >> 1) + (size_t)((cv.col_offset + n) >> 1);
  const uint32_t w0 = (uint32_t)__half_as_ushort(h[0]) | ((uint32_t)__half_as_ushort(h[1]) << 16);
  const uint32_t w1 = (uint32_t)__half_as_ushort(h[2]) | ((uint32_t)__half_as_ushort(h[3]) << 16);
  for (int r = 0; r < cv.world; ++r) {
    uint2* dst = reinterpret_cast<uint2*>(cv.bufs[r] + cv.gather_off) + word;
    if (n + 1 < n_out) tp_st_word(dst, w0, ep);
    if (n + 3 < n_out) tp_st_word(dst + 1, w1, ep);
  }
}

}  // namespace uniql
