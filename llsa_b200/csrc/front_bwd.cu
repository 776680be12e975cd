// Backward of what stands in front of the attention operators: the 2-D rotation of q and k and their RMSNorm
// (models/rope_dit_transformer_2d.py:215-238 run backwards), both tensors in one launch.
//
//   g  = rotation^-1 (dy), every product and sum rounded to the element type as rope_kernel<..., BWD> does (rope.cu)
//   dx = rstd * (g w - xh * mean(g w xh)),  dw = sum over rows of g xh,   xh = x rstd,  rstd = rsqrt(mean(x^2) + eps)
//
// HBM-bound: reads dy and x, writes dx (dx may be dy's own memory).  A CTA takes chunks of fb_rows * (threads / lanes)
// neighbouring tokens of one (b,h) slice, so the slice is found once per chunk and every thread has all its loads (row of dy, of x,
// of the table) in flight before it uses one.  The weight gradient is kept in registers over all chunks of a CTA, reduced through
// shared memory, and leaves as one [C] row per CTA; a one-CTA-per-tensor kernel adds the rows in order (bit-reproducible).
// B=4 H=6 N=16384, [B,N,H,D] storage, both tensors: 302 MB in 63 us = 4.8 TB/s; the rotation's two launches and the eager fp32 formula it
// replaces took 2050 us.  Instructions come next after the memory (0.6 a scheduler and cycle): channels are taken in pairs (66 us one by one); the next
// chunk's rows in flight early, in registers at three CTAs per SM or by cp.async at four, cost more instructions than they hide time (79 and 77 us), and five
// CTAs per SM spill or leave the loads too few registers (65.5).
#include <string.h>

#include <type_traits>

#include "common.cuh"
#include "mma_frag.cuh"

namespace llsa {

constexpr int kFbThreads = 256, kFbC = 64;

template <typename T>
struct FrontBwdArgs {
  View<const T> dy[2], x[2];
  View<T> dx[2];
  const float* w[2];       // fp32 [C] or nullptr (ones)
  float* dw_partial;       // [tensor][gridDim.x][C] or nullptr
  const void* freq;        // [S, C] (even columns sin, odd columns cos) or nullptr
  int64_t fs;
  float eps;
  int norm_mask;
  int H, chunks_per_head;
  int S, n_chunks;
};

// Rows a thread takes at a time: with the norm two keep the registers at four CTAs per SM (four rows: 128 registers, two CTAs, 94 us
// at the size above), without it four.
constexpr int fb_rows(bool norm) { return norm ? 2 : 4; }

template <typename T>
__device__ __forceinline__ void unpack16(const uint4& x, float (&v)[16 / sizeof(T)]) {
  if constexpr (sizeof(T) == 4) {
    v[0] = __uint_as_float(x.x); v[1] = __uint_as_float(x.y); v[2] = __uint_as_float(x.z); v[3] = __uint_as_float(x.w);
  } else {
    v[0] = bf16_lo(x.x); v[1] = bf16_hi(x.x); v[2] = bf16_lo(x.y); v[3] = bf16_hi(x.y);
    v[4] = bf16_lo(x.z); v[5] = bf16_hi(x.z); v[6] = bf16_lo(x.w); v[7] = bf16_hi(x.w);
  }
}
template <typename T>
__device__ __forceinline__ uint4 pack16(const float (&v)[16 / sizeof(T)]) {
  if constexpr (sizeof(T) == 4) return make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
  else return make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
}

// g of one 16-byte group after the inverse rotation by table entries f.  bf16 data with a bf16 table in packed arithmetic: the sum or
// product of two bf16 values rounded to fp32 and then to bf16 is the value rounded once (24 >= 2 * 8 + 2 bits).
__device__ __forceinline__ uint32_t unrotate_pair(uint32_t g, uint32_t f) {       // (cos ge + sin go, -sin ge + cos go)
  const uint32_t cc = __byte_perm(f, 0u, 0x3232), ss = __byte_perm(f, 0u, 0x1010) ^ 0x80000000u, sw = __byte_perm(g, 0u, 0x1032);
  const __nv_bfloat162 x = __hmul2_rn(*reinterpret_cast<const __nv_bfloat162*>(&cc), *reinterpret_cast<const __nv_bfloat162*>(&g)),
                       y = __hmul2_rn(*reinterpret_cast<const __nv_bfloat162*>(&ss), *reinterpret_cast<const __nv_bfloat162*>(&sw));
  const __nv_bfloat162 z = __hadd2_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&z);
}
template <typename T, typename TF>
__device__ __forceinline__ void unrotate(uint4& raw, const TF* fp) {
  if constexpr (sizeof(T) == 2 && sizeof(TF) == 2) {
    const uint4 f = *reinterpret_cast<const uint4*>(fp);
    raw = make_uint4(unrotate_pair(raw.x, f.x), unrotate_pair(raw.y, f.y), unrotate_pair(raw.z, f.z), unrotate_pair(raw.w, f.w));
  } else {
    using P = typename std::conditional<(sizeof(TF) > sizeof(T)), TF, T>::type;      // products and sums are rounded to the wider type
    constexpr int VEC = 16 / sizeof(T);
    float g[VEC], f[VEC];
    unpack16<T>(raw, g);
#pragma unroll
    for (int i = 0; i < VEC; i += 16 / (int) sizeof(TF)) {
      float part[16 / sizeof(TF)];
      unpack16<TF>(*reinterpret_cast<const uint4*>(fp + i), part);
#pragma unroll
      for (int j = 0; j < 16 / (int) sizeof(TF); ++j) f[i + j] = part[j];
    }
#pragma unroll
    for (int j = 0; j < VEC; j += 2) {
      const float sn = f[j], cs = f[j + 1], ge = g[j], go = g[j + 1];
      g[j] = round_to<P>(__fadd_rn(round_to<P>(__fmul_rn(cs, ge)), round_to<P>(__fmul_rn(sn, go))));
      g[j + 1] = round_to<P>(__fadd_rn(round_to<P>(__fmul_rn(-sn, ge)), round_to<P>(__fmul_rn(cs, go))));
    }
    raw = pack16<T>(g);
  }
}

// T: element type of the data, TF: of the table
template <typename T, typename TF, bool NORM>
__global__ void __launch_bounds__(kFbThreads, NORM ? 4 : 1) front_bwd_kernel(FrontBwdArgs<T> a) {
  constexpr int VEC = 16 / sizeof(T), LANES = kFbC / VEC, STEP = kFbThreads / LANES, ROWS = fb_rows(NORM);
  const int ti = blockIdx.y, r0 = threadIdx.x / LANES, c = (threadIdx.x % LANES) * VEC;
  const bool norm = NORM && ((a.norm_mask >> ti) & 1);
  const TF* freq = reinterpret_cast<const TF*>(a.freq);
  pdl_wait();
  F2 w[VEC / 2], dw2[VEC / 2];          // channels in pairs: one instruction for two
#pragma unroll
  for (int i = 0; i < VEC / 2; ++i) {
    w[i] = norm && a.w[ti] ? f2(a.w[ti][c + 2 * i], a.w[ti][c + 2 * i + 1]) : f2(1.f, 1.f);
    dw2[i] = f2(0.f, 0.f);
  }
  for (int ch = blockIdx.x; ch < a.n_chunks; ch += gridDim.x) {
    const int bh = ch / a.chunks_per_head, s0 = (ch - bh * a.chunks_per_head) * (STEP * ROWS) + r0;
    const int b = bh / a.H, h = bh - b * a.H;
    const T* dyp = a.dy[ti].head(b, h) + c;
    const T* xp = NORM ? a.x[ti].head(b, h) + c : nullptr;
    T* dxp = a.dx[ti].head(b, h) + c;
    uint4 g[ROWS], x[ROWS];
#pragma unroll
    for (int u = 0; u < ROWS; ++u) {     // rows past the end are computed on the last row (the reductions need every lane) and dropped
      const int64_t s = min(s0 + u * STEP, a.S - 1);
      g[u] = *reinterpret_cast<const uint4*>(dyp + s * a.dy[ti].sn);
      if (NORM) if (norm) x[u] = *reinterpret_cast<const uint4*>(xp + s * a.x[ti].sn);
    }
#pragma unroll
    for (int u = 0; u < ROWS; ++u) {
      const int s = s0 + u * STEP;
      if (freq) unrotate<T, TF>(g[u], freq + (int64_t) min(s, a.S - 1) * a.fs + c);
      if (NORM) {
        if (norm) {
          float gv[VEC], xv[VEC];
          unpack16<T>(g[u], gv);
          unpack16<T>(x[u], xv);
          F2 gw[VEC / 2], ss2 = f2(0.f, 0.f), dot2 = ss2;
#pragma unroll
          for (int i = 0; i < VEC / 2; ++i) {
            const F2 xi = f2(xv[2 * i], xv[2 * i + 1]);
            gw[i] = f2_mul(f2(gv[2 * i], gv[2 * i + 1]), w[i]);
            ss2 = f2_fma(xi, xi, ss2);
            dot2 = f2_fma(gw[i], xi, dot2);
          }
          float ss, dot, ss1, dot1;
          f2_get(ss2, ss, ss1);
          f2_get(dot2, dot, dot1);
          ss += ss1;
          dot += dot1;
#pragma unroll
          for (int o = 1; o < LANES; o <<= 1) {
            ss += __shfl_xor_sync(0xffffffffu, ss, o);
            dot += __shfl_xor_sync(0xffffffffu, dot, o);
          }
          const float rstd = rsqrtf(ss / (float) kFbC + a.eps), k = dot * rstd / (float) kFbC;      // k = mean(g w xh)
          // rstd meets x before it meets k and itself again: without an eps the square of it leaves the range of a float long before dx does.  (Kernel alone, in a
          // graph, B=4 H=6 N=16384: with the square 65.5 us, so 65.9, with k rstd beside x rstd 66.7.)
          const float live = s < a.S ? rstd : 0.f;
          const F2 l2 = f2(live, live), k2 = f2(-k, -k);
#pragma unroll
          for (int i = 0; i < VEC / 2; ++i) {
            const F2 xh = f2_mul(f2(xv[2 * i], xv[2 * i + 1]), l2);
            dw2[i] = f2_fma(f2(gv[2 * i], gv[2 * i + 1]), xh, dw2[i]);
            f2_get(f2_mul(f2_fma(xh, k2, gw[i]), l2), gv[2 * i], gv[2 * i + 1]);
          }
          g[u] = pack16<T>(gv);
        }
      }
      if (s < a.S) *reinterpret_cast<uint4*>(dxp + (int64_t) s * a.dx[ti].sn) = g[u];
    }
  }
  if (NORM && a.dw_partial) {
    __shared__ float sw[kFbThreads / 32][kFbC];
    const int warp = threadIdx.x >> 5;
    float dw[VEC];
#pragma unroll
    for (int i = 0; i < VEC / 2; ++i) f2_get(dw2[i], dw[2 * i], dw[2 * i + 1]);
#pragma unroll
    for (int i = 0; i < VEC; ++i)
#pragma unroll
      for (int o = LANES; o < 32; o <<= 1) dw[i] += __shfl_xor_sync(0xffffffffu, dw[i], o);
    if ((threadIdx.x & 31) < LANES)
#pragma unroll
      for (int i = 0; i < VEC; ++i) sw[warp][c + i] = dw[i];
    __syncthreads();
    if (threadIdx.x < kFbC) {
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < kFbThreads / 32; ++k) s += sw[k][threadIdx.x];
      a.dw_partial[((int64_t) ti * gridDim.x + blockIdx.x) * kFbC + threadIdx.x] = s;
    }
  }
}

// dw[ti][c] = sum over the CTAs' rows, 16 strided partial sums per channel added in order
__global__ void __launch_bounds__(1024) front_dw_kernel(const float* __restrict__ partial, int rows, float* dw0, float* dw1) {
  pdl_trigger();
  pdl_wait();
  __shared__ float sm[16][kFbC];
  const int c = threadIdx.x & 63, k = threadIdx.x >> 6;
  const float* p = partial + (int64_t) blockIdx.x * rows * kFbC + c;
  float s = 0.f;
#pragma unroll 10
  for (int r = k; r < rows; r += 16) s += p[(int64_t) r * kFbC];
  sm[k][c] = s;
  __syncthreads();
  if (k == 0) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) t += sm[i][c];
    float* out = blockIdx.x == 0 ? dw0 : dw1;
    if (out) out[c] = t;
  }
}

constexpr int kFbMaxCtas = 148 * 4;

template <typename T, typename TF>
static int launch_front_bwd(int n, FrontBwdArgs<T>& a, int64_t BH, int grid, cudaStream_t st) {
  const dim3 g((unsigned) grid, (unsigned) n);
  // The launch is made ready while the kernel in front still runs.  (That kernel does not let it begin early: its CTAs would settle unevenly in the end of it,
  // one wave of them, 602 -> 618 us for the layer with norms at B=4 H=6 N=16384.)  Launched plainly: one level, B=4 H=6 N=4096 183.0 instead of 179.6 us,
  // two levels with norms, B=1 H=6 N=16384 209.5 / 207.1.
  if (a.norm_mask) launch_pdl(front_bwd_kernel<T, TF, true>, g, kFbThreads, 0, st, a);
  else launch_pdl(front_bwd_kernel<T, TF, false>, g, kFbThreads, 0, st, a);
  LLSA_LAUNCH_OK("front_bwd_kernel");
  return LLSA_OK;
}

template <typename T>
static int front_bwd_typed(int n, const LlsaTensor* dy, const LlsaTensor* x, const LlsaTensor* const* norm_weight, int norm_mask, float eps,
                           const LlsaTensor* freq, const LlsaTensor* dx, const LlsaTensor* dw_partial, const LlsaTensor* const* dw,
                           cudaStream_t st) {
  FrontBwdArgs<T> a;
  memset(&a, 0, sizeof(a));
  for (int i = 0; i < n; ++i) {
    a.dy[i] = make_view<const T>(&dy[i]);
    a.dx[i] = make_view<T>(&dx[i]);
    if (norm_mask) a.x[i] = make_view<const T>(&x[i]);
    if (norm_weight && norm_weight[i]) a.w[i] = (const float*) norm_weight[i]->ptr;
  }
  a.freq = freq ? freq->ptr : nullptr;
  a.fs = freq ? freq->stride[0] : 0;
  a.eps = eps;
  a.norm_mask = norm_mask;
  a.H = (int) dy[0].shape[1];
  a.S = (int) dy[0].shape[2];
  const int64_t BH = dy[0].shape[0] * dy[0].shape[1];
  const int rows = fb_rows(norm_mask != 0) * kFbThreads / (kFbC * (int) sizeof(T) / 16);
  a.chunks_per_head = (a.S + rows - 1) / rows;
  const int64_t chunks = BH * a.chunks_per_head;
  LLSA_REQUIRE(chunks < (1ll << 31), LLSA_ERR_SHAPE, "rms_rope_bwd: too many rows");
  a.n_chunks = (int) chunks;
  // With norms one wave of four CTAs per SM over all tensors, and as many rows of partial weight gradients for the kernel behind it to add: two waves
  // took the layer with norms and rotation, B=4 H=6 N=16384, 634 us instead of 630.  Without, more and shorter CTAs even out better (rotation, B=4 H=6
  // N=4096: 186.5 us, 187.6 with half as many).
  const int64_t resident = norm_mask ? kFbMaxCtas / n : kFbMaxCtas;
  const int grid = (int) (chunks < resident ? chunks : resident);
  const bool want_dw = norm_mask && dw && (dw[0] || (n > 1 && dw[1]));
  a.dw_partial = want_dw ? (float*) dw_partial->ptr : nullptr;
  int rc;
  if (freq && freq->dtype == LLSA_F32) rc = launch_front_bwd<T, float>(n, a, BH, grid, st);
  else rc = launch_front_bwd<T, T>(n, a, BH, grid, st);
  if (rc || !want_dw) return rc;
  launch_pdl(front_dw_kernel, n, 1024, 0, st, a.dw_partial, grid, dw[0] ? (float*) dw[0]->ptr : nullptr, n > 1 && dw[1] ? (float*) dw[1]->ptr : nullptr);
  LLSA_LAUNCH_OK("front_dw_kernel");
  return LLSA_OK;
}

}  // namespace llsa

using namespace llsa;

extern "C" int64_t llsa_rms_rope_bwd_partial_elems(int n_tensors) { return n_tensors > 0 ? (int64_t) n_tensors * kFbMaxCtas * kFbC : 0; }

extern "C" int llsa_rms_rope_bwd(int n_tensors, const LlsaTensor* dy, const LlsaTensor* x, const LlsaTensor* const* norm_weight, int norm_mask,
                                 float eps, const LlsaTensor* freq, const LlsaTensor* dx, const LlsaTensor* dw_partial,
                                 const LlsaTensor* const* dw, void* stream) {
  LLSA_REQUIRE(dy && dx, LLSA_ERR_NULL, "rms_rope_bwd: null tensor list");
  LLSA_REQUIRE(n_tensors >= 1 && n_tensors <= 2, LLSA_ERR_ARG, "rms_rope_bwd: n_tensors must be 1 or 2");
  LLSA_REQUIRE(norm_mask >= 0 && norm_mask < (1 << n_tensors) && (!norm_mask || x), LLSA_ERR_ARG, "rms_rope_bwd: bad norm mask");
  LLSA_REQUIRE(eps >= 0.f, LLSA_ERR_ARG, "rms_rope_bwd: eps must not be negative");
  const int dt = dy[0].dtype;
  LLSA_REQUIRE(is_float_dtype(dt), LLSA_ERR_DTYPE, "rms_rope_bwd: dtype must be f32 or bf16");
  LLSA_REQUIRE(dy[0].ndim == 4 && dy[0].shape[3] == kFbC, LLSA_ERR_SHAPE, "rms_rope_bwd: tensors must be [B,H,S,64]");
  const int64_t B = dy[0].shape[0], H = dy[0].shape[1], S = dy[0].shape[2], C = kFbC;
  LLSA_REQUIRE(S < (1ll << 31) - 4096, LLSA_ERR_SHAPE, "rms_rope_bwd: S=%lld too long", (long long) S);
  int rc;
  for (int i = 0; i < n_tensors; ++i) {
    if ((rc = check_bhnd(&dy[i], "dy", dt, B, H, S, C))) return rc;
    if ((rc = check_bhnd(&dx[i], "dx", dt, B, H, S, C))) return rc;
    if (!((norm_mask >> i) & 1)) continue;
    if ((rc = check_bhnd(&x[i], "x", dt, B, H, S, C))) return rc;
    const int64_t sw[1] = {C};
    if (norm_weight && norm_weight[i] && (rc = check_contig(norm_weight[i], "norm weight", LLSA_F32, 1, sw))) return rc;
    if (dw && dw[i]) {
      if ((rc = check_contig(dw[i], "dw", LLSA_F32, 1, sw))) return rc;
      LLSA_REQUIRE(dw_partial && dw_partial->ptr && dw_partial->dtype == LLSA_F32 && dw_partial->ndim == 1 && is_contiguous(dw_partial) &&
                       dw_partial->shape[0] >= llsa_rms_rope_bwd_partial_elems(n_tensors),
                   LLSA_ERR_WORKSPACE, "rms_rope_bwd: dw_partial scratch missing or too small");
    }
  }
  if (freq) {
    LLSA_REQUIRE(freq->ptr && freq->ndim == 2 && freq->shape[0] == S && freq->shape[1] == C && freq->stride[1] == 1, LLSA_ERR_SHAPE,
                 "rms_rope_bwd: freq must be [S,64] with unit inner stride");
    LLSA_REQUIRE(freq->dtype == dt || freq->dtype == LLSA_F32, LLSA_ERR_DTYPE, "rms_rope_bwd: the table must be f32 or have the dtype of the data");
    LLSA_REQUIRE(((uintptr_t) freq->ptr % 16) == 0 && (freq->stride[0] * (int64_t) dtype_size(freq->dtype)) % 16 == 0, LLSA_ERR_STRIDE,
                 "rms_rope_bwd: table rows must be 16-byte aligned");
  }
  if (B * H * S == 0) return LLSA_OK;
  cudaStream_t st = (cudaStream_t) stream;
  return dt == LLSA_F32 ? front_bwd_typed<float>(n_tensors, dy, x, norm_weight, norm_mask, eps, freq, dx, dw_partial, dw, st)
                        : front_bwd_typed<__nv_bfloat16>(n_tensors, dy, x, norm_weight, norm_mask, eps, freq, dx, dw_partial, dw, st);
}
