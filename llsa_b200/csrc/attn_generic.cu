// Plain-FFMA attention kernels for any supported dtype (fp32 and bf16).
//
// They round to the tensor dtype where the reference's kernels do (P before P@V, dS before dS@K; q*scale and k*scale are exact: the
// scale is a power of two), and serve fp32 tensors -- for which the tensor-core kernels do not apply -- as well as bf16 operands outside
// those kernels' limits and a cross-check of the bf16 tensor-core path.
//   attn_fwd_generic   : sparse_attention_res_1.py:9-120 / res_2.py:9-163
//   attn_dq_generic    : preprocess (res_1.py:153-177) + the dQ half of
//                        _attn_bwd_res_dqkv (res_1.py:225-281, res_2.py:287-369)
//   attn_dkv_generic   : the dK/dV half via the CSR (res_1.py:283-327) and the
//                        pooled-key gradients (res_1.py:330-400, res_2.py:418-575)
//
// A CTA owns one 16-row block (queries; keys for dK/dV) and its eight warps share out the 16-row blocks it meets, a block pair per
// warp: the chain of a block's list is an eighth as long, which is what small problems are made of, and no barrier sits between two
// pairs.  Lane (a, b) = (lane / 4, lane % 4) of a warp owns rows a and a + 8:
//   scores     s[i][j] = A[a + 8 i] . B[b + 4 j], six 128-bit shared loads (rows padded to 68 floats: no conflicts) per 32 FMAs
//   accumulate acc[i][4 j + c] += p(a + 8 i, kk) X[kk][16 j + 4 b + c]: p comes from the lane that owns it (shuffle), four loads per 32 FMAs
// so the FMA pipe, not shared memory, is the bound of large problems.  The warps' partial results meet in shared memory in warp order
// (bit-reproducible).  One CTA of 128 threads per block with two scalar shared loads per FMA took 28 (forward), 37 (dQ), 62 (pooled dK/dV)
// and 132 us (fine dK/dV) at B=1 H=2 N=1024 fp32; this form 10, 11, 16 and 29.
#include <string.h>

#include "attn.cuh"

namespace llsa {

constexpr int kGw = 8;                     // warps per CTA
constexpr int kLd = kD + 4;                // padded shared-memory row, floats
constexpr int kTileF = kBS * kLd;          // floats of a staged 16 x 64 tile

// 16 rows x 64 channels by one warp, converted to fp32
template <typename T>
__device__ __forceinline__ void stage_tile(float* dst, const T* src, int64_t stride, int lane) {
  const int r0 = lane >> 4, c = (lane & 15) * 4;
  float4 v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const T* p = src + (int64_t) (2 * i + r0) * stride + c;
    if constexpr (sizeof(T) == 2) {
      const uint2 x = __ldg(reinterpret_cast<const uint2*>(p));
      v[i] = make_float4(bf16_lo(x.x), bf16_hi(x.x), bf16_lo(x.y), bf16_hi(x.y));
    } else {
      v[i] = __ldg(reinterpret_cast<const float4*>(p));
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) *reinterpret_cast<float4*>(dst + (2 * i + r0) * kLd + c) = v[i];
}

__device__ __forceinline__ void tile_scores(float (&s)[2][4], const float* A, const float* B, int a, int b) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
  for (int d = 0; d < kD; d += 4) {
    float4 x[2], y[4];
#pragma unroll
    for (int i = 0; i < 2; ++i) x[i] = *reinterpret_cast<const float4*>(A + (a + 8 * i) * kLd + d);
#pragma unroll
    for (int j = 0; j < 4; ++j) y[j] = *reinterpret_cast<const float4*>(B + (b + 4 * j) * kLd + d);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = fmaf(x[i].x, y[j].x, s[i][j]); s[i][j] = fmaf(x[i].y, y[j].y, s[i][j]);
        s[i][j] = fmaf(x[i].z, y[j].z, s[i][j]); s[i][j] = fmaf(x[i].w, y[j].w, s[i][j]);
      }
  }
}

__device__ __forceinline__ void tile_accumulate(float (&acc)[2][16], const float (&p)[2][4], const float* X, int lane) {
  const int b = lane & 3;
#pragma unroll
  for (int kk = 0; kk < kBS; ++kk) {
    const int src = (lane & ~3) | (kk & 3);
    const float p0 = __shfl_sync(0xffffffffu, p[0][kk >> 2], src), p1 = __shfl_sync(0xffffffffu, p[1][kk >> 2], src);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 x = *reinterpret_cast<const float4*>(X + kk * kLd + 16 * j + 4 * b);
      acc[0][4 * j] = fmaf(p0, x.x, acc[0][4 * j]); acc[0][4 * j + 1] = fmaf(p0, x.y, acc[0][4 * j + 1]);
      acc[0][4 * j + 2] = fmaf(p0, x.z, acc[0][4 * j + 2]); acc[0][4 * j + 3] = fmaf(p0, x.w, acc[0][4 * j + 3]);
      acc[1][4 * j] = fmaf(p1, x.x, acc[1][4 * j]); acc[1][4 * j + 1] = fmaf(p1, x.y, acc[1][4 * j + 1]);
      acc[1][4 * j + 2] = fmaf(p1, x.z, acc[1][4 * j + 2]); acc[1][4 * j + 3] = fmaf(p1, x.w, acc[1][4 * j + 3]);
    }
  }
}

__device__ __forceinline__ void acc_zero(float (&acc)[2][16]) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int d = 0; d < 16; ++d) acc[i][d] = 0.f;
}
// the accumulator of a warp as a [16][kLd] tile
__device__ __forceinline__ void acc_park(float* tile, const float (&acc)[2][16], int lane) {
  const int a = lane >> 2, b = lane & 3;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      *reinterpret_cast<float4*>(tile + (a + 8 * i) * kLd + 16 * j + 4 * b) =
          make_float4(acc[i][4 * j], acc[i][4 * j + 1], acc[i][4 * j + 2], acc[i][4 * j + 3]);
}
__device__ __forceinline__ float quad4_max(float v) {
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
  return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
}
__device__ __forceinline__ float quad4_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}
template <typename T>
__device__ __forceinline__ void store4(T* p, float x, float y, float z, float w) {
  if constexpr (sizeof(T) == 2) *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(x, y), pack_bf16(z, w));
  else *reinterpret_cast<float4*>(p) = make_float4(x, y, z, w);
}

// Resolves key block `i` of the concatenated list [fine | pooled-1 | pooled-2] of a query block.
template <typename T>
__device__ __forceinline__ void key_block(const AttnP<T>& a, int64_t b, int64_t h, int64_t bh, int64_t qb, int i, const T*& kp,
                                          const T*& vp, int64_t& ks, int64_t& vs, float& w, float& kvw) {
  if (i < a.topk) {
    const int64_t j = fine_block(a, bh, qb, i);
    kp = a.k.row(b, h, j * kBS); vp = a.v.row(b, h, j * kBS); ks = a.k.sn; vs = a.v.sn; w = 1.f; kvw = 1.f;
  } else if (i < a.topk + a.p1_blocks) {
    const int64_t j = p1_block(a, bh, qb, i - a.topk);
    kp = a.pk + (bh * a.n1 + j * kBS) * kD; vp = a.pv + (bh * a.n1 + j * kBS) * kD; ks = vs = kD; w = a.w1; kvw = a.kvw1;
  } else {
    const int64_t j = i - a.topk - a.p1_blocks;
    kp = a.pk2 + (bh * a.n2 + j * kBS) * kD; vp = a.pv2 + (bh * a.n2 + j * kBS) * kD; ks = vs = kD; w = a.w2; kvw = a.kvw2;
  }
}

// dynamic shared memory: two [16][kLd] tiles of the CTA's own block, then two per warp
constexpr size_t kGenericSmem = (size_t) (2 + 2 * kGw) * kTileF * sizeof(float);

template <typename T>
__global__ void __launch_bounds__(kGw * 32) attn_fwd_generic(AttnP<T> a) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  __shared__ float s_m[kGw][kBS], s_l[kGw][kBS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ra = lane >> 2, rb = lane & 3;
  const int64_t qb = blockIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
  float *qs = sm, *ks = sm + (2 + 2 * warp) * kTileF, *vs = ks + kTileF;
  if (warp == 0) stage_tile<T>(qs, a.q.row(b, h, qb * kBS), a.q.sn, lane);
  __syncthreads();
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, acc[2][16];
  acc_zero(acc);
  const int nblk = a.topk + a.p1_blocks + a.p2_blocks;
  for (int i = warp; i < nblk; i += kGw) {
    const T *kp, *vp;
    int64_t kst, vst;
    float w, kvw;
    key_block(a, b, h, bh, qb, i, kp, vp, kst, vst, w, kvw);
    __syncwarp();
    stage_tile<T>(ks, kp, kst, lane);
    stage_tile<T>(vs, vp, vst, lane);
    __syncwarp();
    float s[2][4];
    tile_scores(s, qs, ks, ra, rb);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
#pragma unroll
      for (int j = 0; j < 4; ++j) s[r][j] *= a.scale;
      const float mnew = fmaxf(m[r], quad4_max(fmaxf(fmaxf(s[r][0], s[r][1]), fmaxf(s[r][2], s[r][3]))));
      // a warp may meet nothing but scores of -inf (keys masked by the type's lowest value): they weigh 0 whatever the reference
      const float ref = mnew == -INFINITY ? 0.f : mnew;
      const float alpha = expf(m[r] - ref);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[r][j] = expf(s[r][j] - ref);
        sum += s[r][j];
        s[r][j] = round_to<T>(s[r][j]) * w;         // exp_scores.to(v.dtype)
      }
      l[r] = l[r] * alpha + quad4_sum(sum) * w;
      m[r] = mnew;
#pragma unroll
      for (int d = 0; d < 16; ++d) acc[r][d] *= alpha;
    }
    tile_accumulate(acc, s, vs, lane);
  }
  __syncwarp();
  acc_park(ks, acc, lane);
  if (rb == 0) {
#pragma unroll
    for (int r = 0; r < 2; ++r) { s_m[warp][ra + 8 * r] = m[r]; s_l[warp][ra + 8 * r] = l[r]; }
  }
  __syncthreads();
  // thread: four channels of one row
  const int r = threadIdx.x >> 4, c = (threadIdx.x & 15) * 4;
  float mm = -INFINITY, ll = 0.f, o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int u = 0; u < kGw; ++u) mm = fmaxf(mm, s_m[u][r]);
#pragma unroll
  for (int u = 0; u < kGw; ++u) {
    const float f = s_m[u][r] == -INFINITY ? 0.f : expf(s_m[u][r] - mm);
    const float4 x = *reinterpret_cast<const float4*>(sm + (2 + 2 * u) * kTileF + r * kLd + c);
    ll = fmaf(s_l[u][r], f, ll);
    o[0] = fmaf(x.x, f, o[0]); o[1] = fmaf(x.y, f, o[1]); o[2] = fmaf(x.z, f, o[2]); o[3] = fmaf(x.w, f, o[3]);
  }
  store4<T>(a.o.row(b, h, qb * kBS + r) + c, o[0] / ll, o[1] / ll, o[2] / ll, o[3] / ll);
  if (c == 0) a.lse[bh * a.Nq + qb * kBS + r] = mm + logf(ll);
}

template <typename T>
__global__ void __launch_bounds__(kGw * 32) attn_dq_generic(AttnP<T> a) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  __shared__ float s_delta[kBS], s_lse[kBS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ra = lane >> 2, rb = lane & 3;
  const int64_t qb = blockIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
  float *qs = sm, *dos = sm + kTileF, *ks = sm + (2 + 2 * warp) * kTileF, *vs = ks + kTileF;
  if (warp == 0) stage_tile<T>(qs, a.q.row(b, h, qb * kBS), a.q.sn, lane);
  if (warp == 1) stage_tile<T>(dos, a.d_o.row(b, h, qb * kBS), a.d_o.sn, lane);
  __syncthreads();
  {      // delta = rowsum(o * do): sixteen lanes per row
    const int r = threadIdx.x >> 4, c = (threadIdx.x & 15) * 4;
    const T* op = a.o_in.row(b, h, qb * kBS + r) + c;
    float part = 0.f;
#pragma unroll
    for (int d = 0; d < 4; ++d) part = fmaf(to_f32<T>(op[d]), dos[r * kLd + c + d], part);
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if (c == 0) {
      s_delta[r] = part;
      s_lse[r] = a.lse[bh * a.Nq + qb * kBS + r];
      a.delta[bh * a.Nq + qb * kBS + r] = part;
    }
  }
  __syncthreads();
  const float delta[2] = {s_delta[ra], s_delta[ra + 8]}, lse[2] = {s_lse[ra], s_lse[ra + 8]};
  float acc[2][16];
  acc_zero(acc);
  const int nblk = a.topk + a.p1_blocks + a.p2_blocks;
  for (int i = warp; i < nblk; i += kGw) {
    const T *kp, *vp;
    int64_t kst, vst;
    float w, kvw;
    key_block(a, b, h, bh, qb, i, kp, vp, kst, vst, w, kvw);
    __syncwarp();
    stage_tile<T>(ks, kp, kst, lane);
    stage_tile<T>(vs, vp, vst, lane);
    __syncwarp();
    float s[2][4], dp[2][4];
    tile_scores(s, qs, ks, ra, rb);
    tile_scores(dp, dos, vs, ra, rb);
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = expf(s[r][j] * a.scale - lse[r]) * w;
        s[r][j] = round_to<T>(p * (dp[r][j] - delta[r]));       // ds.to(k.dtype)
      }
    tile_accumulate(acc, s, ks, lane);
  }
  __syncwarp();
  acc_park(ks, acc, lane);
  __syncthreads();
  const int r = threadIdx.x >> 4, c = (threadIdx.x & 15) * 4;
  float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int u = 0; u < kGw; ++u) {
    const float4 x = *reinterpret_cast<const float4*>(sm + (2 + 2 * u) * kTileF + r * kLd + c);
    o[0] += x.x; o[1] += x.y; o[2] += x.z; o[3] += x.w;
  }
  store4<T>(a.dq.row(b, h, qb * kBS + r) + c, o[0] * a.scale, o[1] * a.scale, o[2] * a.scale, o[3] * a.scale);
}

// MODE 0: fine KV block blockIdx.x of head blockIdx.y, query blocks from the CSR; writes dk/dv.
// MODE 1: pooled key tile blockIdx.x of query group blockIdx.z (16 query blocks); atomically
//         accumulates into the fp32 pooled-gradient buffers.
// Lane rows are KEYS here (scores are S^T), the columns query rows.
template <typename T, int MODE>
__global__ void __launch_bounds__(kGw * 32) attn_dkv_generic(AttnP<T> a) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ra = lane >> 2, rb = lane & 3;
  const int64_t bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
  float *ks = sm, *vs = sm + kTileF, *qs = sm + (2 + 2 * warp) * kTileF, *dos = qs + kTileF;
  const T *kp, *vp;
  int64_t kst, vst;
  float w = 1.f;
  int64_t list0 = 0, list1 = 0, grp = 0;
  float *gk = nullptr, *gv = nullptr;
  if (MODE == 0) {
    const int64_t j = blockIdx.x;
    kp = a.k.row(b, h, j * kBS); vp = a.v.row(b, h, j * kBS); kst = a.k.sn; vst = a.v.sn;
    if (a.off64) {
      list0 = reinterpret_cast<const int64_t*>(a.offsets)[bh * (a.n1 + 1) + j];
      list1 = reinterpret_cast<const int64_t*>(a.offsets)[bh * (a.n1 + 1) + j + 1];
    } else {
      list0 = reinterpret_cast<const int32_t*>(a.offsets)[bh * (a.n1 + 1) + j];
      list1 = reinterpret_cast<const int32_t*>(a.offsets)[bh * (a.n1 + 1) + j + 1];
    }
    // offsets and list entries handed in by a caller are clamped: nothing is read outside the tensors
    const int64_t E = a.nq1 * a.topk;
    list0 = list0 < 0 ? 0 : (list0 > E ? E : list0);
    list1 = list1 < list0 ? list0 : (list1 > E ? E : list1);
  } else {
    grp = blockIdx.z;
    const int i = blockIdx.x;  // pooled tile of this group: [pooled-1 | pooled-2]
    float wq;
    key_block(a, b, h, bh, grp * kBS, a.topk + i, kp, vp, kst, vst, wq, w);
    const int64_t row0 = (kp - (i < a.p1_blocks ? a.pk : a.pk2)) ;  // element offset of the tile inside its pooled tensor
    gk = (i < a.p1_blocks ? a.dpk : a.dpk2) + row0;
    gv = (i < a.p1_blocks ? a.dpv : a.dpv2) + row0;
    list0 = 0; list1 = kBS;
  }
  if (warp == 0) stage_tile<T>(ks, kp, kst, lane);
  if (warp == 1) stage_tile<T>(vs, vp, vst, lane);
  __syncthreads();
  float dk[2][16], dv[2][16];
  acc_zero(dk);
  acc_zero(dv);
  for (int64_t it = list0 + warp; it < list1; it += kGw) {
    int64_t qb = MODE == 0 ? (int64_t) a.flat[bh * a.nq1 * a.topk + it] : grp * kBS + it;
    qb = qb < 0 ? 0 : (qb >= a.nq1 ? a.nq1 - 1 : qb);
    __syncwarp();
    stage_tile<T>(qs, a.q.row(b, h, qb * kBS), a.q.sn, lane);
    stage_tile<T>(dos, a.d_o.row(b, h, qb * kBS), a.d_o.sn, lane);
    float lse[4], delta[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      lse[j] = a.lse[bh * a.Nq + qb * kBS + rb + 4 * j];
      delta[j] = a.delta[bh * a.Nq + qb * kBS + rb + 4 * j];
    }
    __syncwarp();
    float p[2][4], ds[2][4];
    tile_scores(p, ks, qs, ra, rb);
    tile_scores(ds, vs, dos, ra, rb);
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float x = expf(p[r][j] * a.scale - lse[j]) * w;
        p[r][j] = round_to<T>(x);
        ds[r][j] = round_to<T>(x * (ds[r][j] - delta[j]));
      }
    tile_accumulate(dv, p, dos, lane);
    tile_accumulate(dk, ds, qs, lane);
  }
  __syncwarp();
  acc_park(qs, dk, lane);
  acc_park(dos, dv, lane);
  __syncthreads();
  const int r = threadIdx.x >> 4, c = (threadIdx.x & 15) * 4;
  float sk[4] = {0.f, 0.f, 0.f, 0.f}, sv[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int u = 0; u < kGw; ++u) {
    const float4 x = *reinterpret_cast<const float4*>(sm + (2 + 2 * u) * kTileF + r * kLd + c);
    const float4 y = *reinterpret_cast<const float4*>(sm + (3 + 2 * u) * kTileF + r * kLd + c);
    sk[0] += x.x; sk[1] += x.y; sk[2] += x.z; sk[3] += x.w;
    sv[0] += y.x; sv[1] += y.y; sv[2] += y.z; sv[3] += y.w;
  }
#pragma unroll
  for (int d = 0; d < 4; ++d) sk[d] *= a.scale;
  if (MODE == 0) {
    const int64_t j = blockIdx.x;
    if (a.fold) {
      // pooling backward folded in: dk += (dpk[j] + dpk2[j/16]/16) / 16  (mean_pool.py:54-58 applied twice)
      const float* g1k = a.dpk + (bh * a.n1 + j) * kD + c;
      const float* g1v = a.dpv + (bh * a.n1 + j) * kD + c;
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        float ek = g1k[d], ev = g1v[d];
        if (a.two_level) {
          ek += a.dpk2[(bh * a.n2 + j / kBS) * kD + c + d] * (1.f / kBS);
          ev += a.dpv2[(bh * a.n2 + j / kBS) * kD + c + d] * (1.f / kBS);
        }
        sk[d] += ek * (1.f / kBS);
        sv[d] += ev * (1.f / kBS);
      }
    }
    store4<T>(a.dk.row(b, h, j * kBS + r) + c, sk[0], sk[1], sk[2], sk[3]);
    store4<T>(a.dv.row(b, h, j * kBS + r) + c, sv[0], sv[1], sv[2], sv[3]);
  } else {
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      atomicAdd(gk + r * kD + c + d, sk[d]);
      atomicAdd(gv + r * kD + c + d, sv[d]);
    }
  }
}

template <typename T>
static int fwd_generic_t(const LlsaAttnArgs* g, cudaStream_t st) {
  AttnP<T> a = build_attn_params<T>(g, false);
  dim3 grid((unsigned) a.nq1, (unsigned) (g->q->shape[0] * a.H));
  LLSA_SMEM_LIMIT((attn_fwd_generic<T>), kGenericSmem);
  launch_pdl(attn_fwd_generic<T>, grid, kGw * 32, kGenericSmem, st, a);
  LLSA_LAUNCH_OK("attn_fwd_generic");
  return LLSA_OK;
}

int zero_pooled_acc(const LlsaAttnArgs* g, cudaStream_t st) {
  const int64_t BH = g->q->shape[0] * g->q->shape[1], n1 = g->k->shape[2] / kBS, n2 = n1 / kBS;
  // accumulators that the caller carved out of one allocation, back to back, are cleared by one memset
  char* ptr[4] = {(char*) g->dpk_acc->ptr, (char*) g->dpv_acc->ptr, g->pk2 ? (char*) g->dpk2_acc->ptr : nullptr,
                  g->pk2 ? (char*) g->dpv2_acc->ptr : nullptr};
  const size_t len[4] = {(size_t) BH * n1 * kD * 4, (size_t) BH * n1 * kD * 4, (size_t) BH * n2 * kD * 4, (size_t) BH * n2 * kD * 4};
  for (int i = 0; i < 4;) {
    if (!ptr[i]) { ++i; continue; }
    size_t run = len[i];
    int j = i + 1;
    while (j < 4 && ptr[j] == ptr[i] + run) run += len[j++];
    LLSA_CUDA_OK(cudaMemsetAsync(ptr[i], 0, run, st));
    i = j;
  }
  return LLSA_OK;
}

template <typename T>
static int bwd_generic_t(const LlsaAttnArgs* g, cudaStream_t st) {
  AttnP<T> a = build_attn_params<T>(g, true);
  const unsigned BH = (unsigned) (g->q->shape[0] * a.H);
  const int mask = g->stage_mask ? g->stage_mask : 7;
  if (mask & 1) {
    if (!(g->stage_mask & 8)) {
      int rc = zero_pooled_acc(g, st);
      if (rc) return rc;
    }
    LLSA_SMEM_LIMIT((attn_dq_generic<T>), kGenericSmem);
    launch_pdl(attn_dq_generic<T>, dim3((unsigned) a.nq1, BH), kGw * 32, kGenericSmem, st, a);
    LLSA_LAUNCH_OK("attn_dq_generic");
  }
  const int ptiles = a.p1_blocks + a.p2_blocks;
  if ((mask & 2) && ptiles > 0) {
    LLSA_SMEM_LIMIT((attn_dkv_generic<T, 1>), kGenericSmem);
    launch_pdl(attn_dkv_generic<T, 1>, dim3((unsigned) ptiles, BH, (unsigned) (a.nq1 / kBS)), kGw * 32, kGenericSmem, st, a);
    LLSA_LAUNCH_OK("attn_dkv_generic<pooled>");
  }
  if (mask & 4) {
    LLSA_SMEM_LIMIT((attn_dkv_generic<T, 0>), kGenericSmem);
    launch_pdl(attn_dkv_generic<T, 0>, dim3((unsigned) a.n1, BH), kGw * 32, kGenericSmem, st, a);
    LLSA_LAUNCH_OK("attn_dkv_generic<fine>");
  }
  return LLSA_OK;
}

int launch_attn_fwd_generic(const LlsaAttnArgs* g, cudaStream_t st) {
  return g->q->dtype == LLSA_F32 ? fwd_generic_t<float>(g, st) : fwd_generic_t<__nv_bfloat16>(g, st);
}
int launch_attn_bwd_generic(const LlsaAttnArgs* g, cudaStream_t st) {
  return g->q->dtype == LLSA_F32 ? bwd_generic_t<float>(g, st) : bwd_generic_t<__nv_bfloat16>(g, st);
}

}  // namespace llsa
