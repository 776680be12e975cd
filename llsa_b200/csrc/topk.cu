// Coarse-to-fine top-k block selection (reference: src/llsa/kernel/triton/topk.py).
//
// coarse_topk_kernel / coarse_topk_mma_kernel (bf16 on the tensor cores)
//                     = gen_sparse_indices (topk.py:6-9): scores pq.pk^T rounded to
//   the input dtype (torch.matmul writes its result in the input dtype), then the
//   top-k columns per row, descending.  The score matrix never leaves the SM: a CTA
//   owns ROWS query rows, streams the keys in chunks through shared memory and
//   carries the running top-k list from chunk to chunk.
// refine_topk_kernel  = compute_topk_indices_sparse (topk.py:102-197): one CTA per
//   level-2 query block scores its bs query rows against the bs*p_topk children of
//   the selected parents in fp32 (not rounded, topk.py:141-143).
// Both pick winners by repeated arg-max with ties going to the smallest index, the
// rule the reference's own kernels use (topk.py:60-62, :159-161).
#include <math_constants.h>

#include "common.cuh"
#include "mma_frag.cuh"
#include "topk_words.cuh"

namespace llsa {

constexpr int kMaxTopk = 64;

struct Cand {
  float v;
  int64_t i;
};

__device__ __forceinline__ bool better(float v2, int64_t i2, float v, int64_t i) { return v2 > v || (v2 == v && i2 < i); }

// Scores as the selection sees them: a NaN score ranks as the largest value (torch.topk's order, so a row of
// NaNs still yields topk distinct in-range columns); NaN is thereby free to mark "retired / unused" entries,
// which `better` never prefers.
__device__ __forceinline__ float nan_first(float v) { return v != v ? CUDART_INF_F : v; }

__device__ __forceinline__ Cand warp_argmax(Cand c) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float v2 = __shfl_xor_sync(0xffffffffu, c.v, o);
    const int64_t i2 = __shfl_xor_sync(0xffffffffu, c.i, o);
    if (better(v2, i2, c.v, c.i)) { c.v = v2; c.i = i2; }
  }
  return c;
}

template <typename T>
__device__ __forceinline__ float dot_row(const float* __restrict__ q, const T* __restrict__ k, int D) {
  float acc = 0.f;
  if constexpr (sizeof(T) == 2) {
    for (int d = 0; d < D; d += 8) {
      uint4 x = ldg128(k + d);
      acc = fmaf(q[d], bf16_lo(x.x), acc); acc = fmaf(q[d + 1], bf16_hi(x.x), acc);
      acc = fmaf(q[d + 2], bf16_lo(x.y), acc); acc = fmaf(q[d + 3], bf16_hi(x.y), acc);
      acc = fmaf(q[d + 4], bf16_lo(x.z), acc); acc = fmaf(q[d + 5], bf16_hi(x.z), acc);
      acc = fmaf(q[d + 6], bf16_lo(x.w), acc); acc = fmaf(q[d + 7], bf16_hi(x.w), acc);
    }
  } else {
    for (int d = 0; d < D; d += 4) {
      float4 x = __ldg(reinterpret_cast<const float4*>(k + d));
      acc = fmaf(q[d], x.x, acc); acc = fmaf(q[d + 1], x.y, acc); acc = fmaf(q[d + 2], x.z, acc); acc = fmaf(q[d + 3], x.w, acc);
    }
  }
  return acc;
}

constexpr int kCoarseRows = 8;
constexpr int kCoarseChunk = 1024;
constexpr int kCoarseThreads = 128;

// pq, pk: contiguous [B*H, M|n, D].  idx out: [B*H, M, topk] int32 or int64.
template <typename T>
__global__ void __launch_bounds__(kCoarseThreads)
coarse_topk_kernel(const T* __restrict__ pq, const T* __restrict__ pk, void* __restrict__ idx_out, int idx64, int64_t M, int64_t n, int D,
                   int topk) {
  extern __shared__ float sm[];
  float* qs = sm;                                   // [ROWS][D]
  float* sc = qs + kCoarseRows * D;                 // [ROWS][CHUNK]
  float* cv = sc + kCoarseRows * kCoarseChunk;      // [ROWS][kMaxTopk] carried values
  int64_t* ci = reinterpret_cast<int64_t*>(cv + kCoarseRows * kMaxTopk);  // carried indices
  float* nv = reinterpret_cast<float*>(ci + kCoarseRows * kMaxTopk);      // [ROWS][kMaxTopk] next list
  int64_t* ni = reinterpret_cast<int64_t*>(nv + kCoarseRows * kMaxTopk);

  const int64_t bh = blockIdx.y;
  const int64_t row0 = (int64_t) blockIdx.x * kCoarseRows;
  const int nrows = (int) min((int64_t) kCoarseRows, M - row0);
  const T* q0 = pq + (bh * M + row0) * D;
  const T* k0 = pk + bh * n * D;
  for (int i = threadIdx.x; i < kCoarseRows * D; i += blockDim.x) qs[i] = (i / D) < nrows ? to_f32<T>(q0[i]) : 0.f;
  for (int i = threadIdx.x; i < kCoarseRows * kMaxTopk; i += blockDim.x) { cv[i] = CUDART_NAN_F; ci[i] = INT64_MAX; }
  __syncthreads();

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  for (int64_t base = 0; base < n; base += kCoarseChunk) {
    const int cn = (int) min((int64_t) kCoarseChunk, n - base);
    for (int j = threadIdx.x; j < cn; j += blockDim.x) {
      const T* kr = k0 + (base + j) * D;
#pragma unroll
      for (int r = 0; r < kCoarseRows; ++r) sc[r * kCoarseChunk + j] = nan_first(round_to<T>(dot_row<T>(qs + r * D, kr, D)));
    }
    __syncthreads();
    for (int r = warp; r < nrows; r += nwarps) {
      float* s = sc + r * kCoarseChunk;
      for (int t = 0; t < topk; ++t) {
        Cand best{-CUDART_INF_F, INT64_MAX};
        for (int j = lane; j < cn; j += 32) {
          const float v = s[j];
          if (better(v, base + j, best.v, best.i)) { best.v = v; best.i = base + j; }
        }
        if (lane < topk) {
          const float v = cv[r * kMaxTopk + lane];
          const int64_t i = ci[r * kMaxTopk + lane];
          if (better(v, i, best.v, best.i)) { best.v = v; best.i = i; }
        }
        if (topk > 32 && lane + 32 < topk) {
          const float v = cv[r * kMaxTopk + lane + 32];
          const int64_t i = ci[r * kMaxTopk + lane + 32];
          if (better(v, i, best.v, best.i)) { best.v = v; best.i = i; }
        }
        best = warp_argmax(best);
        if (lane == 0) { nv[r * kMaxTopk + t] = best.v; ni[r * kMaxTopk + t] = best.i; }
        // retire the winner from whichever set holds it
        if (best.i >= base && best.i < base + cn) {
          if (lane == 0) s[best.i - base] = CUDART_NAN_F;
        } else {
          for (int u = lane; u < topk; u += 32)
            if (ci[r * kMaxTopk + u] == best.i) cv[r * kMaxTopk + u] = CUDART_NAN_F;
        }
        __syncwarp();
      }
      for (int u = lane; u < topk; u += 32) { cv[r * kMaxTopk + u] = nv[r * kMaxTopk + u]; ci[r * kMaxTopk + u] = ni[r * kMaxTopk + u]; }
      __syncwarp();
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < nrows * topk; i += blockDim.x) {
    const int r = i / topk, t = i % topk;
    const int64_t o = (bh * M + row0 + r) * topk + t;
    const int64_t v = ci[r * kMaxTopk + t];
    if (idx64) reinterpret_cast<int64_t*>(idx_out)[o] = v;
    else reinterpret_cast<int32_t*>(idx_out)[o] = (int32_t) v;
  }
}

// ---- coarse selection on the tensor cores (bf16, D = 64, top-k <= 8) ---------------------------
// Scores are rounded to bf16 as torch.matmul would store them (topk.py:7), so a score and its column fit one 32-bit word:
// the order-preserving image of the bf16 value above the complemented column (65535 - column).  Larger word = better candidate,
// ties already decided in favour of the smaller column, and a candidate list is kept sorted with integer minima and maxima.
//   * A warp owns ROWT * 16 query rows (the m16 of mma.sync.m16n8k16) and every KW-th 16-key block; its key fragments come straight
//     from L1 / L2 (one 256-bit load per lane and eight keys), the next block's while this one is scored.
//   * Lists of 1024 keys and more: pass 1 scores all keys and keeps the maximum of each lane's columns per row.  The top-k-th largest
//     of a row's 4 KW group maxima bounds its top-k-th score from below (with 16 groups some eleven scores of a row reach it,
//     whatever its length).  Pass 2 scores the keys again and looks only at what reaches the bound: a quarter of the instructions per
//     score, and few insertions.  Without a bound the kernel spends its time inserting: until a lane has seen most of its columns, some
//     lane of the warp has something to insert in almost every block (235 us below).  A bound from every fourth block leaves
//     four times as many insertions (158 us); below 1024 keys the two barriers cost what the bound saves.
//   * The row's 4 KW sorted lists meet in shared memory: lane l holds list l, a round takes the largest head, its owner moves on.
// Large problems are bound by the latency of a warp's product and comparison chains (four warps per scheduler, tensor pipe 41 % busy);
// keys through a cp.async ring or 24 warps per SM of one row tile each changed nothing.  n = M = 4096, 8 slices: 243 us with one pass
// and lists of (value, column) pairs in four-warp CTAs of 64 rows, 139 now; n = M = 1024, 8 slices: 59 -> 20; n = M = 256, 24
// slices: 24 -> 6.7; n = M = 64, 6 slices: 14.9 -> 3.7.  Long lists are topk_tc.cu's.
constexpr int kCmWarps = 8, kCmBoundFrom = 1024;

// ROWT row tiles per warp, KW warps share a CTA's keys, the other kCmWarps / KW are further row tiles.
template <int ROWT, int KW>
__global__ void __launch_bounds__(kCmWarps * 32)
coarse_topk_mma_kernel(const bf16* __restrict__ pq, const bf16* __restrict__ pk, void* __restrict__ idx_out, int idx64, int64_t M, int64_t n,
                       int topk) {
  pdl_trigger();
  pdl_wait();
  constexpr int RG = kCmWarps / KW, ROWS = RG * ROWT * 16;
  __shared__ uint32_t lists[ROWS][KW * 4 * kCmTop + 4];      // + 4: rows shift by four banks.  Pass 1: the group maxima
  __shared__ uint32_t bound[ROWS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int kw = warp % KW, wrow = (warp / KW) * ROWT * 16;
  const int64_t bh = blockIdx.y, row0 = (int64_t) blockIdx.x * ROWS + wrow;
  const bf16* k0 = pk + bh * n * 64;
  const int n_blk = (int) (n / 16);
  RowFrag q[ROWT][2];
#pragma unroll
  for (int r = 0; r < ROWT; ++r) {                            // rows past M are computed and dropped
    load_rowfrag(q[r][0], pq + (bh * M + min(row0 + r * 16 + g, M - 1)) * 64, t);
    load_rowfrag(q[r][1], pq + (bh * M + min(row0 + r * 16 + g + 8, M - 1)) * 64, t);
  }
  // scores of this warp's blocks, one after the other: visit(block number, scores)
  auto walk = [&](auto&& visit) {
    RowFrag ka, kb;
    if (kw < n_blk) {
      load_rowfrag(ka, k0 + (int64_t) (kw * 16 + g) * 64, t);
      load_rowfrag(kb, k0 + (int64_t) (kw * 16 + 8 + g) * 64, t);
    }
    for (int blk = kw; blk < n_blk; blk += KW) {
      float s[ROWT][2][4];
#pragma unroll
      for (int r = 0; r < ROWT; ++r) mma_rows_x_keys_z(s[r][0], s[r][1], q[r][0], q[r][1], ka, kb);
      if (blk + KW < n_blk) {
        const int c = (blk + KW) * 16;
        load_rowfrag(ka, k0 + (int64_t) (c + g) * 64, t);
        load_rowfrag(kb, k0 + (int64_t) (c + 8 + g) * 64, t);
      }
      visit(blk, s);
    }
  };
  // ---- pass 1: group maxima -> bounds
  const bool bounded = n >= kCmBoundFrom;
  if (bounded) {
    float m[ROWT][2];
#pragma unroll
    for (int r = 0; r < ROWT; ++r) m[r][0] = m[r][1] = -CUDART_INF_F;
    walk([&](int, const float (&s)[ROWT][2][4]) {
#pragma unroll
      for (int r = 0; r < ROWT; ++r)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          m[r][e] = fmax3(fmax3(m[r][e], s[r][0][2 * e], s[r][0][2 * e + 1]), s[r][1][2 * e], s[r][1][2 * e + 1]);
    });
#pragma unroll
    for (int r = 0; r < ROWT; ++r)
#pragma unroll
      for (int e = 0; e < 2; ++e) {                      // no column, or none but -inf and NaN: 0, no bound
        uint32_t w, other;
        candidate_words(m[r][e], 0.f, 0u, w, other);
        lists[wrow + r * 16 + g + 8 * e][kw * 4 + t] = m[r][e] > -CUDART_INF_F ? w & 0xFFFF0000u : 0u;
      }
    __syncthreads();
    for (int r = warp; r < ROWS; r += kCmWarps) {
      uint32_t x = lane < KW * 4 ? lists[r][lane] : 0u, best = 0u;
      for (int u = 0; u < topk; ++u) {
        best = __reduce_max_sync(0xffffffffu, x);
        const unsigned who = __ballot_sync(0xffffffffu, x == best);
        if (lane == __ffs((int) who) - 1) x = 0u;
      }
      if (lane == 0) bound[r] = best;
    }
    __syncthreads();
  }
  // ---- pass 2: what reaches the bound
  uint32_t list[ROWT][2][kCmTop], thr[ROWT][2];
  float low[ROWT][2];          // a score below this rounds to less than the bound
#pragma unroll
  for (int r = 0; r < ROWT; ++r)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      bound_limits(bounded ? bound[wrow + r * 16 + g + 8 * e] : 0u, thr[r][e], low[r][e]);
#pragma unroll
      for (int u = 0; u < kCmTop; ++u) list[r][e][u] = 0u;
    }
  walk([&](int blk, const float (&s)[ROWT][2][4]) {
    const uint32_t c = (uint32_t) (blk * 16 + 2 * t), inv0 = (65535u - c) | ((65534u - c) << 16), inv1 = inv0 - 0x00080008u;
#pragma unroll
    for (int r = 0; r < ROWT; ++r)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (max_nan(max_nan(s[r][0][2 * e], s[r][0][2 * e + 1]), max_nan(s[r][1][2 * e], s[r][1][2 * e + 1])) < low[r][e]) continue;      // false for NaN
        uint32_t k[4];
        candidate_words(s[r][0][2 * e], s[r][0][2 * e + 1], inv0, k[0], k[1]);
        candidate_words(s[r][1][2 * e], s[r][1][2 * e + 1], inv1, k[2], k[3]);
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (k[u] > thr[r][e]) {
            list_insert(list[r][e], k[u]);
            thr[r][e] = umax(thr[r][e], list[r][e][kCmTop - 1]);
          }
      }
  });
#pragma unroll
  for (int r = 0; r < ROWT; ++r)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int u = 0; u < kCmTop; ++u) lists[wrow + r * 16 + g + 8 * e][(kw * 4 + t) * kCmTop + u] = list[r][e][u];
  __syncthreads();
  for (int r = warp; r < ROWS; r += kCmWarps) {
    const int64_t row = (int64_t) blockIdx.x * ROWS + r;
    if (row >= M) continue;
    const uint32_t* mine = &lists[r][lane * kCmTop];
    uint32_t head = lane < KW * 4 ? mine[0] : 0u, won = 0u;
    int at = 0;
    for (int u = 0; u < topk; ++u) {
      const uint32_t best = __reduce_max_sync(0xffffffffu, head);
      if (lane == u) won = best;
      if (head == best) { ++at; head = at < kCmTop ? mine[at] : 0u; }      // candidate words are distinct: one owner
    }
    if (lane < topk) {
      const int64_t o = (bh * M + row) * topk + lane;
      const uint32_t col = 65535u - (won & 0xFFFFu);
      if (idx64) reinterpret_cast<int64_t*>(idx_out)[o] = (int64_t) col;
      else reinterpret_cast<int32_t*>(idx_out)[o] = (int32_t) col;
    }
  }
}

// ---- coarse selection with scalar arithmetic, D = 64, top-k <= 32 (fp32, and the bf16 shapes below) ------------------------
// A score is one fp32 chain over the channels in order, so fp32 and the bf16 shapes that were always scored this way (list
// lengths that are no multiple of 64, top-k above 8) keep their scores bit for bit.  A CTA owns 16 query rows and walks the keys in
// chunks of 256 through shared memory; a thread scores 8 rows x 2 keys (64 FMAs per sixteen 128-bit shared loads: FMA and shared
// pipes are in balance).  A row's running list lives in a warp, sorted, one candidate per lane; only candidates above its
// last entry cost more than a comparison.  One thread per key and eight rows one after the other, with a scan over all scores per
// winner (coarse_topk_kernel below, kept for other D and longer lists), took 18 us at n = M = 64, B H = 2 (fp32), 32 us at
// n = M = 160, top-16, B H = 5 and 4850 us at n = M = 4064, B H = 8; this form 10.5, 18 and 865.
constexpr int kCtRows = 16, kCtKeys = 256, kCtPitch = 68, kCtScPitch = kCtKeys + 4;
constexpr size_t kCtSmem = ((size_t) (kCtRows + kCtKeys) * kCtPitch + (size_t) kCtRows * kCtScPitch) * 4;

__device__ __forceinline__ uint32_t orderable(float v);

// Sorted list of the best `topk` 64-bit candidates (score image above the complemented column) spread over a warp, lane u holding
// the u-th; `thr` is the last one.  Every lane brings one candidate (0: none).
__device__ __forceinline__ void warp_list_insert(uint64_t& list, uint64_t& thr, uint64_t cand, int topk, int lane) {
  unsigned todo = __ballot_sync(0xffffffffu, cand > thr);
  while (todo) {
    const uint64_t c = __shfl_sync(0xffffffffu, cand, __ffs((int) todo) - 1);
    const int pos = __popc(__ballot_sync(0xffffffffu, list > c));
    const uint64_t up = __shfl_up_sync(0xffffffffu, list, 1);
    list = lane == pos ? c : (lane > pos ? up : list);
    thr = __shfl_sync(0xffffffffu, list, topk - 1);
    todo &= (todo - 1) & __ballot_sync(0xffffffffu, cand > thr);
  }
}

template <typename T>
__device__ __forceinline__ float4 load4(const T* p) {
  if constexpr (sizeof(T) == 2) {
    const uint2 x = __ldg(reinterpret_cast<const uint2*>(p));
    return make_float4(bf16_lo(x.x), bf16_hi(x.x), bf16_lo(x.y), bf16_hi(x.y));
  } else {
    return __ldg(reinterpret_cast<const float4*>(p));
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
coarse_topk_tile_kernel(const T* __restrict__ pq, const T* __restrict__ pk, void* __restrict__ idx_out, int idx64, int64_t M, int64_t n, int topk) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  float* qs = sm;                                   // [16][kCtPitch]
  float* ks = qs + kCtRows * kCtPitch;              // [256][kCtPitch]
  uint32_t* sc = reinterpret_cast<uint32_t*>(ks + kCtKeys * kCtPitch);      // [16][kCtScPitch] score images
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t bh = blockIdx.y, row0 = (int64_t) blockIdx.x * kCtRows;
  const T* k0 = pk + bh * n * 64;
  {
    const int r = tid >> 4, d = (tid & 15) * 4;
    *reinterpret_cast<float4*>(qs + r * kCtPitch + d) = load4<T>(pq + (bh * M + min(row0 + r, M - 1)) * 64 + d);
  }
  const int rw = (warp >> 2) * 8, kw = (warp & 3) * 64 + lane;      // this thread's rows and its first key
  uint64_t list[2] = {0, 0}, thr[2] = {0, 0};
  for (int64_t base = 0; base < n; base += kCtKeys) {
    const int cn = (int) min((int64_t) kCtKeys, n - base);
    for (int i = tid; i < cn * 16; i += 256) {
      const int r = i >> 4, d = (i & 15) * 4;
      *reinterpret_cast<float4*>(ks + r * kCtPitch + d) = load4<T>(k0 + (base + r) * 64 + d);
    }
    __syncthreads();
    if ((warp & 3) * 64 < cn) {                     // keys past the chunk's end read stale rows and are dropped by the selection
      float acc[8][2];
#pragma unroll
      for (int r = 0; r < 8; ++r) acc[r][0] = acc[r][1] = 0.f;
#pragma unroll 4
      for (int d = 0; d < 64; d += 4) {
        const float4 x = *reinterpret_cast<const float4*>(ks + kw * kCtPitch + d), y = *reinterpret_cast<const float4*>(ks + (kw + 32) * kCtPitch + d);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const float4 q = *reinterpret_cast<const float4*>(qs + (rw + r) * kCtPitch + d);
          acc[r][0] = fmaf(q.x, x.x, acc[r][0]); acc[r][0] = fmaf(q.y, x.y, acc[r][0]);
          acc[r][0] = fmaf(q.z, x.z, acc[r][0]); acc[r][0] = fmaf(q.w, x.w, acc[r][0]);
          acc[r][1] = fmaf(q.x, y.x, acc[r][1]); acc[r][1] = fmaf(q.y, y.y, acc[r][1]);
          acc[r][1] = fmaf(q.z, y.z, acc[r][1]); acc[r][1] = fmaf(q.w, y.w, acc[r][1]);
        }
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        sc[(rw + r) * kCtScPitch + kw] = orderable(nan_first(round_to<T>(acc[r][0])));
        sc[(rw + r) * kCtScPitch + kw + 32] = orderable(nan_first(round_to<T>(acc[r][1])));
      }
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const uint32_t* s = sc + (warp + 8 * e) * kCtScPitch;
      for (int j = lane; j - lane < cn; j += 32) {
        const uint64_t cand = j < cn ? ((uint64_t) s[j] << 32) | (0xFFFFFFFFu - (uint32_t) (base + j)) : 0;
        warp_list_insert(list[e], thr[e], cand, topk, lane);
      }
    }
  }
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int64_t row = row0 + warp + 8 * e;
    if (row < M && lane < topk) {
      const int64_t o = (bh * M + row) * topk + lane;
      const uint32_t col = 0xFFFFFFFFu - (uint32_t) list[e];
      if (idx64) reinterpret_cast<int64_t*>(idx_out)[o] = (int64_t) col;
      else reinterpret_cast<int32_t*>(idx_out)[o] = (int32_t) col;
    }
  }
}

// Refine step.  pq1: contiguous [B*H, M, D] (M query blocks); pk1: contiguous [B*H, Mk, D] (Mk key blocks, Mk != M when the
// queries are a shard of the sequence); p_idx [B*H, M/bs, p_topk] with values in [0, Mk/bs); out [B*H, M, topk].
// MMA = true (bf16, D = 64, bs = 16): the 16 x C score tile comes from mma.sync with fp32
// accumulation of the exact bf16 products, as the reference's tl.dot does.
// Order-preserving map of a float onto uint32 (larger float <=> larger integer, -0 and +0 share one image so
// that they tie like the float comparison does).
__device__ __forceinline__ uint32_t orderable(float v) {
  uint32_t u = __float_as_uint(v);
  if (u == 0x80000000u) u = 0u;
  if (v != v) u = 0x7FC00000u;           // any NaN ranks above +inf, as in torch.topk
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// The best `topk` (at most 32) of up to 256 candidates of each of ROWS rows, lane l holding candidates l, l + 32, ... (eight of them) as 64-bit words: the
// order-preserving image of the score above the complemented index; 0: none.  A lane sorts its words once, so that its best is always slot 0.  A
// round is one warp maximum over the score images and a ballot (a second maximum, over the complemented indices, only where scores tie); the winner's
// lane shifts its list up by one, and winner t stays in lane t of `mine`, complemented.  Two rows at a time: the rounds are chains of warp-wide
// instructions, and two chains hide each other's latency.
template <int ROWS>
__device__ __forceinline__ void select_sorted8(uint64_t (&w)[ROWS][8], uint32_t (&mine)[ROWS], int topk, int lane) {
  constexpr int SLOTS = 8;
#pragma unroll
  for (int e = 0; e < ROWS; ++e) {
    mine[e] = 0u;
#pragma unroll
    for (int k = 2; k <= SLOTS; k <<= 1)                          // bitonic, descending
#pragma unroll
      for (int j = k >> 1; j > 0; j >>= 1)
#pragma unroll
        for (int i = 0; i < SLOTS; ++i)
          if ((i ^ j) > i) {
            const bool desc = (i & k) == 0;
            const uint64_t x = w[e][i], y = w[e][i ^ j];
            const bool sw = desc ? y > x : x > y;
            w[e][i] = sw ? y : x;
            w[e][i ^ j] = sw ? x : y;
          }
  }
  for (int t = 0; t < topk; ++t) {
#pragma unroll
    for (int e = 0; e < ROWS; ++e) {
      const uint32_t hi = (uint32_t) (w[e][0] >> 32), lo = (uint32_t) w[e][0];
      const uint32_t m = __reduce_max_sync(0xffffffffu, hi);
      unsigned who = __ballot_sync(0xffffffffu, hi == m);
      if (who & (who - 1)) {                                      // equal scores: the smallest index
        const uint32_t ml = __reduce_max_sync(0xffffffffu, hi == m ? lo : 0u);
        who = __ballot_sync(0xffffffffu, hi == m && lo == ml);
      }
      const int src = __ffs((int) who) - 1;
      const uint32_t win = __shfl_sync(0xffffffffu, lo, src);
      if (lane == t) mine[e] = win;
      if (lane == src) {                                          // candidates are distinct: one owner
#pragma unroll
        for (int u = 0; u + 1 < SLOTS; ++u) w[e][u] = w[e][u + 1];
        w[e][SLOTS - 1] = 0;
      }
    }
  }
}

// Refine selection of lists of up to 256 candidates; one store writes a row's list (a store by each winner is 20 % slower).
__device__ __forceinline__ void refine_select_sorted8(const float* sc, const int* cand, int C, int bs, int topk, void* idx_out, int idx64,
                                                      int64_t out_row0, int warp, int lane, int nwarps) {
  for (int r0 = warp; r0 < bs; r0 += 2 * nwarps) {
    uint64_t w[2][8];
    uint32_t mine[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float* s = sc + min(r0 + e * nwarps, bs - 1) * C;      // past the last row: computed on it and dropped
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int j = lane + 32 * u;
        w[e][u] = (j < C && cand[j] >= 0) ? ((uint64_t) orderable(s[j]) << 32) | (0xFFFFFFFFu - (uint32_t) cand[j]) : 0;      // 0 is below every real candidate
      }
    }
    select_sorted8<2>(w, mine, topk, lane);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int r = r0 + e * nwarps;
      if (r < bs && lane < topk) {
        const int64_t o = (out_row0 + r) * topk + lane;
        const uint32_t blk = 0xFFFFFFFFu - mine[e];
        if (idx64) reinterpret_cast<int64_t*>(idx_out)[o] = (int64_t) blk;
        else reinterpret_cast<int32_t*>(idx_out)[o] = (int32_t) blk;
      }
    }
  }
}

// The same for at most 128 candidates (four per lane) with 32-bit words, which is faster there (33.0 against 34.3 us at 48 slices of 64
// parents): a lane sorts its four
// candidates once (descending score image, ascending block index among equals), so its best is always slot 0; a round is two warp
// reductions, the winner's lane shifts its list up by one, and winner t stays in lane t until one store writes the row's list.
__device__ __forceinline__ void refine_select_sorted4(const float* sc, const int* cand, int C, int bs, int topk, void* idx_out, int idx64,
                                                      int64_t out_row0, int warp, int lane, int nwarps) {
  for (int r = warp; r < bs; r += nwarps) {
    const float* s = sc + r * C;
    uint32_t key[4], blk[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = lane + 32 * u;
      key[u] = (j < C && cand[j] >= 0) ? orderable(s[j]) : 0u;            // 0 is below every real score's image
      blk[u] = j < C ? (uint32_t) cand[j] : 0xFFFFFFFFu;
    }
    auto order = [&](int x, int y) {                     // afterwards slot x is not worse than slot y
      const bool sw = key[y] > key[x] || (key[y] == key[x] && blk[y] < blk[x]);
      const uint32_t kx = sw ? key[y] : key[x], ky = sw ? key[x] : key[y], bx = sw ? blk[y] : blk[x], by = sw ? blk[x] : blk[y];
      key[x] = kx; key[y] = ky; blk[x] = bx; blk[y] = by;
    };
    order(0, 1); order(2, 3); order(0, 2); order(1, 3); order(1, 2);
    uint32_t mine = 0;                                   // winner number `lane` of this row
    for (int t = 0; t < topk; ++t) {
      const uint32_t mk = __reduce_max_sync(0xffffffffu, key[0]);
      const uint32_t mb = __reduce_min_sync(0xffffffffu, key[0] == mk ? blk[0] : 0xFFFFFFFFu);
      if (key[0] == mk && blk[0] == mb) {               // candidates are distinct blocks: one owner
        key[0] = key[1]; blk[0] = blk[1]; key[1] = key[2]; blk[1] = blk[2]; key[2] = key[3]; blk[2] = blk[3];
        key[3] = 0u; blk[3] = 0xFFFFFFFFu;
      }
      if (lane == t) mine = mb;
    }
    if (lane < topk) {
      const int64_t o = (out_row0 + r) * topk + lane;
      if (idx64) reinterpret_cast<int64_t*>(idx_out)[o] = (int64_t) mine;
      else reinterpret_cast<int32_t*>(idx_out)[o] = (int32_t) mine;
    }
  }
}

// Coarse selection of ONE level-2 query block inside the refine kernel's CTA: against 64 level-2 keys on the tensor cores (four warps: 16 keys
// each).  The scores are the ones coarse_topk_mma_kernel computes -- the same mma.sync k-steps in the same order on the same
// operands (all 16 A rows hold the query block's row, so every row of the result is that row's), rounded to bf16, NaN first --
// and the winners come out in the same order (descending score, ties to the smaller key), so the fused form returns the
// bits of the two-kernel form while saving its launch and its 64 x 64-score CTAs.
struct FusedCoarse {
  const void* pq2;     // [BH, M / bs, 64], the data's type
  const void* pk2;     // [BH, n2, 64]
  void* pidx_out;      // [BH, M / bs, p_topk]
  int pidx64;
};

__device__ __forceinline__ void coarse_row_64(const FusedCoarse& f, int64_t bh, int64_t P, int64_t n2q, int p_topk, float* sc2, int* s_pidx) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  RowFrag q2, ka, kb;
  load_rowfrag(q2, reinterpret_cast<const bf16*>(f.pq2) + (bh * n2q + P) * 64, t);
  const bf16* k0 = reinterpret_cast<const bf16*>(f.pk2) + bh * 64 * 64;
  load_rowfrag(ka, k0 + (warp * 16 + g) * 64, t);
  load_rowfrag(kb, k0 + (warp * 16 + 8 + g) * 64, t);
  float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
  mma_rows_x_keys(s0, s1, q2, q2, ka, kb);
  if (g == 0) {
    const int c = warp * 16 + 2 * t;
    sc2[c] = round_to<bf16>(s0[0]); sc2[c + 1] = round_to<bf16>(s0[1]);
    sc2[c + 8] = round_to<bf16>(s1[0]); sc2[c + 9] = round_to<bf16>(s1[1]);
  }
  __syncthreads();
  if (warp == 0) {
    uint32_t key[2], blk[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      key[u] = orderable(sc2[lane + 32 * u]);
      blk[u] = (uint32_t) (lane + 32 * u);
    }
    uint32_t mine = 0;
    for (int tt = 0; tt < p_topk; ++tt) {
      const uint32_t bk = key[1] > key[0] ? key[1] : key[0];
      const uint32_t bb = key[1] > key[0] ? blk[1] : blk[0];      // equal scores: the smaller key (slot 0) wins
      const uint32_t mk = __reduce_max_sync(0xffffffffu, bk);
      const uint32_t mb = __reduce_min_sync(0xffffffffu, bk == mk ? bb : 0xFFFFFFFFu);
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (blk[u] == mb) { key[u] = 0u; blk[u] = 0xFFFFFFFFu; }
      if (lane == tt) mine = mb;
    }
    if (lane < p_topk) {
      s_pidx[lane] = (int) mine;
      const int64_t o = (bh * n2q + P) * p_topk + lane;
      if (f.pidx64) reinterpret_cast<int64_t*>(f.pidx_out)[o] = (int64_t) mine;
      else reinterpret_cast<int32_t*>(f.pidx_out)[o] = (int32_t) mine;
    }
  }
  __syncthreads();
}

// The same with scalar arithmetic for the level-2 lists coarse_topk_tile_kernel would take (same channel order, same bits), up to
// kFusedKeys keys, one thread per key.
constexpr int kFusedKeys = 256;
template <typename T>
__device__ __forceinline__ void coarse_row_scalar(const FusedCoarse& f, int64_t bh, int64_t P, int64_t n2q, int n2, int p_topk, uint32_t* sc2,
                                                  int* s_pidx) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const T* q = reinterpret_cast<const T*>(f.pq2) + (bh * n2q + P) * 64;
  for (int j = threadIdx.x; j < n2; j += blockDim.x) {
    const T* k = reinterpret_cast<const T*>(f.pk2) + (bh * n2 + j) * 64;
    float acc = 0.f;
#pragma unroll 8
    for (int d = 0; d < 64; d += 4) {
      const float4 a = load4<T>(q + d), x = load4<T>(k + d);
      acc = fmaf(a.x, x.x, acc); acc = fmaf(a.y, x.y, acc); acc = fmaf(a.z, x.z, acc); acc = fmaf(a.w, x.w, acc);
    }
    sc2[j] = orderable(nan_first(round_to<T>(acc)));
  }
  __syncthreads();
  if (warp == 0) {
    uint64_t w[1][8];
    uint32_t mine[1];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int j = lane + 32 * u;
      w[0][u] = j < n2 ? ((uint64_t) sc2[j] << 32) | (0xFFFFFFFFu - (uint32_t) j) : 0;
    }
    select_sorted8<1>(w, mine, p_topk, lane);
    if (lane < p_topk) {
      const uint32_t col = 0xFFFFFFFFu - mine[0];
      s_pidx[lane] = (int) col;
      const int64_t o = (bh * n2q + P) * p_topk + lane;
      if (f.pidx64) reinterpret_cast<int64_t*>(f.pidx_out)[o] = (int64_t) col;
      else reinterpret_cast<int32_t*>(f.pidx_out)[o] = (int32_t) col;
    }
  }
  __syncthreads();
}

// FUSED: 0 parents given, 1 selected here by coarse_row_64, 2 by coarse_row_scalar.
// A CTA is a chain of short steps (parents, keys, scores, rounds of the selection), so what counts is how many of them an SM holds, and that they are few
// waves: PER_SM of them, 9 (8 with the scalar step) where the compiler's choice of registers allowed 8 and 5.  H=5 N=40960, top-16: 49 us with five an SM,
// where 800 CTAs are 740 and a second wave of 60, parents inserted into a list one by one and keys loaded when they are needed; 32.8 now.  Lists of eight
// parents: B=8 H=6 N=16384 31.8 -> 29.9, B=4 19.7 -> 18.6, B=1 8.8 -> 8.2, B=3 H=5 N=5376 10.0 -> 8.9.
template <typename T, bool MMA, int FUSED = 0, int PER_SM = FUSED < 2 ? 9 : 8>
__global__ void __launch_bounds__(128, PER_SM)
refine_topk_kernel(const T* __restrict__ pq1, const T* __restrict__ pk1, IdxView p_idx, void* __restrict__ idx_out, int idx64, int64_t M,
                   int64_t Mk, int D_, int topk, int p_topk, int bs_, FusedCoarse fused) {
  pdl_trigger();
  pdl_wait();
  // constants where the dispatch fixes them: no division by a run-time block size per candidate
  const int D = MMA || FUSED ? 64 : D_, bs = MMA || FUSED ? 16 : bs_;
  extern __shared__ float sm[];
  __shared__ float s_sc2[FUSED == 2 ? kFusedKeys : 64];
  __shared__ int s_pidx[kMaxTopk];
  const int C = p_topk * bs;
  float* qs = sm;                 // [bs][D]
  float* sc = qs + bs * D;        // [bs][C]
  int* cand = reinterpret_cast<int*>(sc + bs * C);  // [C] block index of each candidate
  const int64_t bh = blockIdx.y, P = blockIdx.x, n2q = M / bs, n2 = Mk / bs;
  const T* q0 = pq1 + (bh * M + P * bs) * D;
  const T* k0 = pk1 + bh * Mk * D;
  if constexpr (!MMA)                                    // the tensor-core path takes its query fragments straight from global memory
    for (int i = threadIdx.x; i < bs * D; i += blockDim.x) qs[i] = to_f32<T>(q0[i]);
  if constexpr (FUSED == 1) coarse_row_64(fused, bh, P, n2q, p_topk, s_sc2, s_pidx);
  if constexpr (FUSED == 2) coarse_row_scalar<T>(fused, bh, P, n2q, (int) n2, p_topk, reinterpret_cast<uint32_t*>(s_sc2), s_pidx);
  for (int j = threadIdx.x; j < C; j += blockDim.x) {
    int64_t p = FUSED ? (int64_t) s_pidx[j / bs] : p_idx.at((bh * n2q + P) * p_topk + j / bs);
    p = p < 0 ? 0 : (p >= n2 ? n2 - 1 : p);      // never read outside the tensor
    // a parent listed twice (possible only in a caller-made p_idx) contributes its children once: the selection
    // below relies on distinct candidate blocks; the repeats are marked unused (-1)
    bool repeat = false;
    for (int u = 0; u < j / bs; ++u) {
      int64_t pu = FUSED ? (int64_t) s_pidx[u] : p_idx.at((bh * n2q + P) * p_topk + u);
      pu = pu < 0 ? 0 : (pu >= n2 ? n2 - 1 : pu);
      repeat = repeat || pu == p;
    }
    cand[j] = repeat ? -1 : (int) (p * bs + j % bs);
  }
  __syncthreads();
  if constexpr (MMA) {
    const int warp_ = threadIdx.x >> 5, lane_ = threadIdx.x & 31, g = lane_ >> 2, t = lane_ & 3;
    if constexpr (sizeof(T) == 2) {
      RowFrag qlo, qhi;
      load_rowfrag(qlo, reinterpret_cast<const bf16*>(q0) + g * D, t);
      load_rowfrag(qhi, reinterpret_cast<const bf16*>(q0) + (g + 8) * D, t);
      RowFrag ka, kb;
      auto keys = [&](int tile) {
        load_rowfrag(ka, reinterpret_cast<const bf16*>(k0) + (int64_t) max(cand[tile * 8 + g], 0) * D, t);
        load_rowfrag(kb, reinterpret_cast<const bf16*>(k0) + (int64_t) max(cand[tile * 8 + 8 + g], 0) * D, t);
      };
      if (warp_ * 2 < C / 8) keys(warp_ * 2);
      for (int tile = warp_ * 2; tile < C / 8; tile += 8) {      // two 8-candidate n-tiles per step and warp; the next step's keys on their way
        float s0[4], s1[4];
        mma_rows_x_keys_z(s0, s1, qlo, qhi, ka, kb);
        if (tile + 8 < C / 8) keys(tile + 8);
        // C fragment: rows g / g+8, candidates tile*8 + 2t, +1 (and +8 for the second tile)
        sc[g * C + tile * 8 + 2 * t] = s0[0];       sc[g * C + tile * 8 + 2 * t + 1] = s0[1];
        sc[(g + 8) * C + tile * 8 + 2 * t] = s0[2]; sc[(g + 8) * C + tile * 8 + 2 * t + 1] = s0[3];
        sc[g * C + tile * 8 + 8 + 2 * t] = s1[0];       sc[g * C + tile * 8 + 9 + 2 * t] = s1[1];
        sc[(g + 8) * C + tile * 8 + 8 + 2 * t] = s1[2]; sc[(g + 8) * C + tile * 8 + 9 + 2 * t] = s1[3];
      }
    }
  } else
  // each thread owns a candidate: its key row is read once per group of 16 query rows and
  // meets the rows (broadcast from shared memory) in 16 independent accumulators
  for (int j = threadIdx.x; j < C; j += blockDim.x) {
    const T* kr = k0 + (int64_t) max(cand[j], 0) * D;
    for (int r0 = 0; r0 < bs; r0 += 16) {
      float acc[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) acc[r] = 0.f;
      for (int d = 0; d < D; d += 8) {
        float kv[8];
        if constexpr (sizeof(T) == 2) {
          const uint4 x = ldg128(kr + d);
          kv[0] = bf16_lo(x.x); kv[1] = bf16_hi(x.x); kv[2] = bf16_lo(x.y); kv[3] = bf16_hi(x.y);
          kv[4] = bf16_lo(x.z); kv[5] = bf16_hi(x.z); kv[6] = bf16_lo(x.w); kv[7] = bf16_hi(x.w);
        } else {
          const float4 x = __ldg(reinterpret_cast<const float4*>(kr + d)), y = __ldg(reinterpret_cast<const float4*>(kr + d + 4));
          kv[0] = x.x; kv[1] = x.y; kv[2] = x.z; kv[3] = x.w; kv[4] = y.x; kv[5] = y.y; kv[6] = y.z; kv[7] = y.w;
        }
#pragma unroll
        for (int r = 0; r < 16; ++r) {
          if (r0 + r < bs) {
            const float* qr = qs + (r0 + r) * D + d;
#pragma unroll
            for (int u = 0; u < 8; ++u) acc[r] = fmaf(qr[u], kv[u], acc[r]);
          }
        }
      }
#pragma unroll
      for (int r = 0; r < 16; ++r)
        if (r0 + r < bs) sc[(r0 + r) * C + j] = acc[r];
    }
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  if (C <= 256 && topk <= 32) {
    if (C <= 128) refine_select_sorted4(sc, cand, C, bs, topk, idx_out, idx64, bh * M + P * bs, warp, lane, nwarps);
    else refine_select_sorted8(sc, cand, C, bs, topk, idx_out, idx64, bh * M + P * bs, warp, lane, nwarps);
    return;
  }
  for (int r = warp; r < bs; r += nwarps) {
    float* s = sc + r * C;
    for (int j = lane; j < C; j += 32) s[j] = cand[j] < 0 ? CUDART_NAN_F : nan_first(s[j]);
    __syncwarp();
    for (int t = 0; t < topk; ++t) {
      Cand best{-CUDART_INF_F, INT64_MAX};
      int bj = -1;
      for (int j = lane; j < C; j += 32) {
        const float v = s[j];           // NaN here = retired or a repeated parent's candidate
        if (better(v, cand[j], best.v, best.i)) { best.v = v; best.i = cand[j]; bj = j; }
      }
      const Cand w = warp_argmax(best);
      if (bj >= 0 && w.i == best.i && w.v == best.v) s[bj] = CUDART_NAN_F;  // candidates are distinct blocks: one owner
      if (lane == 0) {
        const int64_t o = (bh * M + P * bs + r) * topk + t;
        if (idx64) reinterpret_cast<int64_t*>(idx_out)[o] = w.i;
        else reinterpret_cast<int32_t*>(idx_out)[o] = (int32_t) w.i;
      }
      __syncwarp();
    }
  }
}

int launch_coarse_topk_tc(const LlsaTensor* pq, const LlsaTensor* pk, const LlsaTensor* idx, int topk, int wait_limit, cudaStream_t st);      // topk_tc.cu

}  // namespace llsa

using namespace llsa;

// The tcgen05 kernel (topk_tc.cu) sums a score in another order, so the length of the list alone may choose between the two: a row's blocks must not depend
// on the batch or on how many of the sequence's rows a call holds.  So the line weighs few rows against many: below it mma.sync is ahead up to eight or twelve
// square slices (n = M), above it tcgen05, its keys shared by a cluster where there are few rows, from three to six on.  us in a graph, smooth inputs,
// here / there: n = 1024: 1 slice 8.8 / 18.4, 6 11.7 / 20.5, 12 21.5 / 25.2, 24 50 / 35, 48 81 / 57; 1536: 1 11.8 / 17.3, 4 14.6 / 24.8, 8 26.5 / 30.2, 16 60 / 42;
// 2048: 1 15.3 / 18.1, 3 17.4 / 24.3, 4 27.4 / 25.1, 8 42.0 / 36.0, 12 72 / 47, 48 217 / 112; 2560: 1 18.3 / 20.6, 2 20.0 / 28.9, 4 33.1 / 36.6, 6 48.7 / 39.2, 12 94 / 48;
// 3072: 2 22.2 / 28.3, 3 36.8 / 37.0, 12 107 / 59; 4096: 1 27.3 / 24.4, 2 45.7 / 34.9, 8 131 / 69, 128 rows 20.0 / 18.6.
constexpr int64_t kCoarseTcFrom = 2048;

// The tensor-core kernel's range: its accumulation order differs from the scalar kernels' in the last bit of a score, so the line
// between the two decides which bits a caller gets and stays where it was (whole 64-key tiles, top-k <= 8).
static bool coarse_on_mma(const LlsaTensor* pq, const LlsaTensor* pk, int topk) {
  const int64_t n = pk->shape[2];
  return pq->dtype == LLSA_BF16 && pq->shape[3] == 64 && topk <= kCmTop && n % 64 == 0 && n <= 65536 && ((uintptr_t) pq->ptr % 32) == 0 &&
         ((uintptr_t) pk->ptr % 32) == 0;
}

extern "C" int llsa_coarse_topk(const LlsaTensor* pq, const LlsaTensor* pk, const LlsaTensor* idx, int topk, void* stream) {
  return llsa_coarse_topk_bounded(pq, pk, idx, topk, 0, stream);
}

extern "C" int llsa_coarse_topk_bounded(const LlsaTensor* pq, const LlsaTensor* pk, const LlsaTensor* idx, int topk, int wait_limit, void* stream) {
  LLSA_REQUIRE(pq && pk && idx && pq->ptr && pk->ptr && idx->ptr, LLSA_ERR_NULL, "coarse_topk: null tensor");
  LLSA_REQUIRE(pq->ndim == 4 && pk->ndim == 4, LLSA_ERR_SHAPE, "coarse_topk: pq, pk must be [B,H,M,D]");
  const int64_t B = pq->shape[0], H = pq->shape[1], M = pq->shape[2], D = pq->shape[3], n = pk->shape[2];
  LLSA_REQUIRE(is_float_dtype(pq->dtype) && pk->dtype == pq->dtype, LLSA_ERR_DTYPE, "coarse_topk: pq/pk must both be f32 or bf16");
  LLSA_REQUIRE(is_index_dtype(idx->dtype), LLSA_ERR_DTYPE, "coarse_topk: idx must be i32 or i64");
  LLSA_REQUIRE(topk >= 1 && topk <= kMaxTopk && topk <= n, LLSA_ERR_ARG, "coarse_topk: topk=%d must be in 1..min(%d, n=%lld)", topk, kMaxTopk, (long long) n);
  LLSA_REQUIRE(D % 8 == 0 && D <= 512, LLSA_ERR_SHAPE, "coarse_topk: D=%lld must be a multiple of 8, at most 512", (long long) D);
  const int64_t sq[4] = {B, H, M, D}, sk[4] = {B, H, n, D}, si[4] = {B, H, M, topk};
  int rc;
  if ((rc = check_contig(pq, "pq", pq->dtype, 4, sq))) return rc;
  if ((rc = check_contig(pk, "pk", pq->dtype, 4, sk))) return rc;
  if ((rc = check_contig(idx, "idx", idx->dtype, 4, si))) return rc;
  if (B * H * M == 0) return LLSA_OK;
  cudaStream_t st = (cudaStream_t) stream;
  const unsigned BH = (unsigned) (B * H);
  const int idx64 = idx->dtype == LLSA_I64;
  const bool bf = pq->dtype == LLSA_BF16;
  auto blocks = [&](int rows) { return dim3((unsigned) ((M + rows - 1) / rows), BH); };
  if (coarse_on_mma(pq, pk, topk) && n >= kCoarseTcFrom) return launch_coarse_topk_tc(pq, pk, idx, topk, wait_limit, st);
  if (coarse_on_mma(pq, pk, topk)) {
    const bf16 *q = (const bf16*) pq->ptr, *k = (const bf16*) pk->ptr;
    // 64 rows per CTA (each key read from L2 once per 64 rows) where that still gives every SM two CTAs, else 16 rows, the keys
    // split over all eight warps
    if (B * H * ((M + 63) / 64) >= 2 * 148) launch_pdl(coarse_topk_mma_kernel<2, 4>, blocks(64), kCmWarps * 32, 0, st, q, k, idx->ptr, idx64, M, n, topk);
    else launch_pdl(coarse_topk_mma_kernel<1, 8>, blocks(16), kCmWarps * 32, 0, st, q, k, idx->ptr, idx64, M, n, topk);
  } else if (D == 64 && topk <= 32 && n < (1ll << 31)) {
    if (bf) {
      LLSA_SMEM_LIMIT((coarse_topk_tile_kernel<bf16>), kCtSmem);
      launch_pdl(coarse_topk_tile_kernel<bf16>, blocks(kCtRows), 256, kCtSmem, st, (const bf16*) pq->ptr, (const bf16*) pk->ptr, idx->ptr, idx64, M, n, topk);
    } else {
      LLSA_SMEM_LIMIT((coarse_topk_tile_kernel<float>), kCtSmem);
      launch_pdl(coarse_topk_tile_kernel<float>, blocks(kCtRows), 256, kCtSmem, st, (const float*) pq->ptr, (const float*) pk->ptr, idx->ptr, idx64, M, n, topk);
    }
  } else {
    const size_t smem = (size_t) kCoarseRows * (D + kCoarseChunk) * 4 + (size_t) kCoarseRows * kMaxTopk * (4 + 8) * 2;
    if (!bf) {
      LLSA_SMEM_LIMIT((coarse_topk_kernel<float>), smem);
      coarse_topk_kernel<float><<<blocks(kCoarseRows), kCoarseThreads, smem, st>>>((const float*) pq->ptr, (const float*) pk->ptr, idx->ptr, idx64, M, n,
                                                                                   (int) D, topk);
    } else {
      LLSA_SMEM_LIMIT((coarse_topk_kernel<bf16>), smem);
      coarse_topk_kernel<bf16><<<blocks(kCoarseRows), kCoarseThreads, smem, st>>>((const bf16*) pq->ptr, (const bf16*) pk->ptr, idx->ptr, idx64, M, n,
                                                                                  (int) D, topk);
    }
  }
  LLSA_LAUNCH_OK("coarse_topk_kernel");
  return LLSA_OK;
}

extern "C" int llsa_refine_topk(const LlsaTensor* pq1, const LlsaTensor* pk1, const LlsaTensor* p_idx, const LlsaTensor* idx, int topk,
                                int p_topk, int block_size, void* stream) {
  LLSA_REQUIRE(pq1 && pk1 && p_idx && idx && pq1->ptr && pk1->ptr && p_idx->ptr && idx->ptr, LLSA_ERR_NULL, "refine_topk: null tensor");
  LLSA_REQUIRE(pq1->ndim == 4 && pk1->ndim == 4, LLSA_ERR_SHAPE, "refine_topk: pq1, pk1 must be [B,H,M,D]");
  const int64_t B = pq1->shape[0], H = pq1->shape[1], M = pq1->shape[2], D = pq1->shape[3], Mk = pk1->shape[2];
  const int bs = block_size;
  LLSA_REQUIRE(is_float_dtype(pq1->dtype) && pk1->dtype == pq1->dtype, LLSA_ERR_DTYPE, "refine_topk: pq1/pk1 must both be f32 or bf16");
  LLSA_REQUIRE(is_index_dtype(idx->dtype) && is_index_dtype(p_idx->dtype), LLSA_ERR_DTYPE, "refine_topk: index tensors must be i32 or i64");
  LLSA_REQUIRE(bs >= 1 && M % bs == 0 && Mk % bs == 0, LLSA_ERR_ARG, "refine_topk: M=%lld / Mk=%lld not divisible by block size %d", (long long) M,
               (long long) Mk, bs);
  LLSA_REQUIRE(p_topk >= 1 && topk >= 1 && topk <= p_topk * bs && p_topk <= Mk / bs, LLSA_ERR_ARG, "refine_topk: bad topk=%d / p_topk=%d", topk, p_topk);
  LLSA_REQUIRE(D % 8 == 0, LLSA_ERR_SHAPE, "refine_topk: D=%lld must be a multiple of 8", (long long) D);
  const size_t smem = ((size_t) bs * D + (size_t) bs * p_topk * bs + (size_t) p_topk * bs) * 4;
  LLSA_REQUIRE(smem <= 200 * 1024, LLSA_ERR_ARG, "refine_topk: bs*p_topk too large");
  const int64_t sq[4] = {B, H, M, D}, sk[4] = {B, H, Mk, D}, sp[4] = {B, H, M / bs, p_topk}, si[4] = {B, H, M, topk};
  int rc;
  if ((rc = check_contig(pq1, "pq1", pq1->dtype, 4, sq))) return rc;
  if ((rc = check_contig(pk1, "pk1", pq1->dtype, 4, sk))) return rc;
  if ((rc = check_contig(p_idx, "p_idx", p_idx->dtype, 4, sp))) return rc;
  if ((rc = check_contig(idx, "idx", idx->dtype, 4, si))) return rc;
  if (B * H * M == 0) return LLSA_OK;
  dim3 grid((unsigned) (M / bs), (unsigned) (B * H));
  cudaStream_t st = (cudaStream_t) stream;
  if (pq1->dtype == LLSA_F32) {
    LLSA_SMEM_LIMIT((refine_topk_kernel<float, false>), smem);
    launch_pdl(refine_topk_kernel<float, false>, grid, 128, smem, st, (const float*) pq1->ptr, (const float*) pk1->ptr, make_idx(p_idx), idx->ptr,
                                                              idx->dtype == LLSA_I64, M, Mk, (int) D, topk, p_topk, bs, FusedCoarse{});
  } else if (D == 64 && bs == 16 && p_topk % 2 == 0 && ((uintptr_t) pq1->ptr % 32) == 0 && ((uintptr_t) pk1->ptr % 32) == 0) {
    LLSA_SMEM_LIMIT((refine_topk_kernel<__nv_bfloat16, true>), smem);
    launch_pdl(refine_topk_kernel<__nv_bfloat16, true>, grid, 128, smem, st, (const __nv_bfloat16*) pq1->ptr, (const __nv_bfloat16*) pk1->ptr,
                                                                     make_idx(p_idx), idx->ptr, idx->dtype == LLSA_I64, M, Mk, (int) D, topk, p_topk, bs, FusedCoarse{});
  } else {
    LLSA_SMEM_LIMIT((refine_topk_kernel<__nv_bfloat16, false>), smem);
    launch_pdl(refine_topk_kernel<__nv_bfloat16, false>, grid, 128, smem, st, (const __nv_bfloat16*) pq1->ptr, (const __nv_bfloat16*) pk1->ptr,
                                                                      make_idx(p_idx), idx->ptr, idx->dtype == LLSA_I64, M, Mk, (int) D, topk, p_topk, bs, FusedCoarse{});
  }
  LLSA_LAUNCH_OK("refine_topk_kernel");
  return LLSA_OK;
}

extern "C" int llsa_select_two_level(const LlsaTensor* pq1, const LlsaTensor* pk1, const LlsaTensor* pq2, const LlsaTensor* pk2,
                                     const LlsaTensor* p_idx, const LlsaTensor* idx, int topk, int p_topk, int block_size, void* stream) {
  LLSA_REQUIRE(pq1 && pk1 && pq2 && pk2 && p_idx && idx, LLSA_ERR_NULL, "select_two_level: null tensor");
  const int bs = block_size;
  // One launch where the level-2 list is short: exactly 64 keys where the tensor-core coarse kernel would score them, or up to
  // kFusedKeys keys where the scalar one would (a CTA then reads the whole level-2 list of its head: 32 KB at most, from L2).
  bool fusable = pq1->ptr && pk1->ptr && pq2->ptr && pk2->ptr && p_idx->ptr && idx->ptr && is_float_dtype(pq1->dtype) && pk1->dtype == pq1->dtype &&
                 pq2->dtype == pq1->dtype && pk2->dtype == pq1->dtype && pq1->ndim == 4 && pk1->ndim == 4 && pq2->ndim == 4 && pk2->ndim == 4 &&
                 pq1->shape[3] == 64 && bs == 16 && p_topk >= 2 && p_topk % 2 == 0 && p_topk <= 16 && p_topk <= pk2->shape[2] &&
                 ((uintptr_t) pq1->ptr % 32) == 0 && ((uintptr_t) pk1->ptr % 32) == 0 && ((uintptr_t) pq2->ptr % 32) == 0 &&
                 ((uintptr_t) pk2->ptr % 32) == 0;
  const bool on_mma = fusable && coarse_on_mma(pq2, pk2, p_topk);
  if (fusable) fusable = on_mma ? pk2->shape[2] == 64 : pk2->shape[2] <= kFusedKeys;
  if (!fusable) {
    int rc = llsa_coarse_topk(pq2, pk2, p_idx, p_topk, stream);
    if (rc) return rc;
    return llsa_refine_topk(pq1, pk1, p_idx, idx, topk, p_topk, block_size, stream);
  }
  const int64_t B = pq1->shape[0], H = pq1->shape[1], M = pq1->shape[2], D = 64, Mk = pk1->shape[2], n2 = pk2->shape[2];
  const int dt = pq1->dtype;
  LLSA_REQUIRE(is_index_dtype(idx->dtype) && is_index_dtype(p_idx->dtype), LLSA_ERR_DTYPE, "select_two_level: index tensors must be i32 or i64");
  LLSA_REQUIRE(M % bs == 0 && Mk == n2 * bs, LLSA_ERR_SHAPE, "select_two_level: M=%lld / Mk=%lld do not fit %lld level-2 keys", (long long) M, (long long) Mk,
               (long long) n2);
  LLSA_REQUIRE(topk >= 1 && topk <= kMaxTopk && topk <= p_topk * bs, LLSA_ERR_ARG, "select_two_level: bad topk=%d / p_topk=%d", topk, p_topk);
  const int64_t sq[4] = {B, H, M, D}, sk[4] = {B, H, Mk, D}, sq2[4] = {B, H, M / bs, D}, sk2[4] = {B, H, n2, D}, sp[4] = {B, H, M / bs, p_topk},
                si[4] = {B, H, M, topk};
  int rc;
  if ((rc = check_contig(pq1, "pq1", dt, 4, sq))) return rc;
  if ((rc = check_contig(pk1, "pk1", dt, 4, sk))) return rc;
  if ((rc = check_contig(pq2, "pq2", dt, 4, sq2))) return rc;
  if ((rc = check_contig(pk2, "pk2", dt, 4, sk2))) return rc;
  if ((rc = check_contig(p_idx, "p_idx", p_idx->dtype, 4, sp))) return rc;
  if ((rc = check_contig(idx, "idx", idx->dtype, 4, si))) return rc;
  if (B * H * M == 0) return LLSA_OK;
  const size_t smem = ((size_t) bs * D + (size_t) bs * p_topk * bs + (size_t) p_topk * bs) * 4;
  FusedCoarse f;
  f.pq2 = pq2->ptr;
  f.pk2 = pk2->ptr;
  f.pidx_out = p_idx->ptr;
  f.pidx64 = p_idx->dtype == LLSA_I64;
  const dim3 grid((unsigned) (M / bs), (unsigned) (B * H));
  cudaStream_t st = (cudaStream_t) stream;
  const int idx64 = idx->dtype == LLSA_I64;
  const IdxView none{nullptr, 0};
  if (dt == LLSA_F32) {
    // Six CTAs per SM cost 48 bytes of spilled registers, five 8: five where they are one wave anyway.  Forward in us, five / six: B=1 H=2 N=4096 (32 CTAs)
    // 45.5 / 46.2, B=3 H=5 N=5376 (315) 290.7 / 292.6, B=1 H=6 N=16384 (384) 425.4 / 426.7; B=2 H=6 N=16384 (768) 855.6 / 851.3, B=1 H=5 N=40960 top-16
    // (800) 1707 / 1702, B=1 H=6 N=65536 (1536) 2458 / 2454.
    auto kernel = B * H * (M / bs) <= 5 * 148 ? refine_topk_kernel<float, false, 2, 5> : refine_topk_kernel<float, false, 2, 6>;
    LLSA_SMEM_LIMIT(kernel, smem);
    launch_pdl(kernel, grid, 128, smem, st, (const float*) pq1->ptr, (const float*) pk1->ptr, none, idx->ptr, idx64, M, Mk, (int) D, topk, p_topk, bs, f);
  } else if (on_mma) {
    LLSA_SMEM_LIMIT((refine_topk_kernel<bf16, true, 1>), smem);
    launch_pdl(refine_topk_kernel<bf16, true, 1>, grid, 128, smem, st, (const bf16*) pq1->ptr, (const bf16*) pk1->ptr, none, idx->ptr, idx64, M, Mk, (int) D, topk,
                                                               p_topk, bs, f);
  } else {
    LLSA_SMEM_LIMIT((refine_topk_kernel<bf16, true, 2>), smem);
    launch_pdl(refine_topk_kernel<bf16, true, 2>, grid, 128, smem, st, (const bf16*) pq1->ptr, (const bf16*) pk1->ptr, none, idx->ptr, idx64, M, Mk, (int) D, topk,
                                                               p_topk, bs, f);
  }
  LLSA_LAUNCH_OK("refine_topk_kernel<fused>");
  return LLSA_OK;
}
