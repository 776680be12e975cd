// Candidates of the coarse selection as 32-bit words, shared by its tensor-core kernels (topk.cu: mma.sync, topk_tc.cu: tcgen05).
// Scores are rounded to bf16 as torch.matmul would store them (topk.py:7), so a score and its column fit one word: the order-preserving image
// of the bf16 value above the complemented column (65535 - column).  Larger word = better candidate, ties already decided in favour of the
// smaller column, words of one row are distinct, and a list of candidates is kept sorted with integer minima and maxima.
#pragma once
#include <math_constants.h>

#include "common.cuh"

namespace llsa {

constexpr int kCmTop = 8;

__device__ __forceinline__ uint32_t umax(uint32_t a, uint32_t b) { return a > b ? a : b; }
__device__ __forceinline__ uint32_t umin(uint32_t a, uint32_t b) { return a < b ? a : b; }

template <uint32_t SEL>
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b) {      // selector bit 3 of a byte: its sign, replicated (__byte_perm drops that bit)
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "n"(SEL));
  return d;
}

// Candidate words of two neighbouring columns: cinv holds 65535 - c (low half) and 65535 - (c + 1) (high half).
// NaN (0x7FFF after the conversion) ranks above everything as in torch.topk, -0 ties with +0.
__device__ __forceinline__ void candidate_words(float s0, float s1, uint32_t cinv, uint32_t& k0, uint32_t& k1) {
  __nv_bfloat162 p = __hadd2(__floats2bfloat162_rn(s0, s1), __float2bfloat162_rn(0.f));      // -0 + 0 = +0
  const uint32_t u = *reinterpret_cast<uint32_t*>(&p);
  const uint32_t o = u ^ (prmt<0xBB99>(u, 0u) | 0x80008000u);      // negative: all bits flipped, else the sign bit set
  k0 = prmt<0x1054>(o, cinv);
  k1 = prmt<0x3276>(o, cinv);
}

__device__ __forceinline__ float max_nan(float a, float b) {      // NaN if either is
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}

__device__ __forceinline__ void list_insert(uint32_t (&list)[kCmTop], uint32_t k) {
  list[kCmTop - 1] = umax(list[kCmTop - 1], k);
#pragma unroll
  for (int u = kCmTop - 1; u > 0; --u) {
    const uint32_t hi = umax(list[u - 1], list[u]), lo = umin(list[u - 1], list[u]);
    list[u - 1] = hi;
    list[u] = lo;
  }
}

// What the bound's word (0: no bound) lets through: `thr`, which a candidate word has to exceed, and `low`, below which a score rounds to less than
// the bound.
__device__ __forceinline__ void bound_limits(uint32_t w, uint32_t& thr, float& low) {
  thr = w > 0u ? w - 1u : 0u;
  const uint32_t below = (w >> 16) - ((w >> 16) == 0x8000u ? 2u : 1u);            // image of the bf16 value one step down (-0 is no step)
  low = w > 0x00800000u ? __uint_as_float((below & 0x8000u ? below ^ 0x8000u : ~below & 0xFFFFu) << 16) : -CUDART_INF_F;
}

}  // namespace llsa
