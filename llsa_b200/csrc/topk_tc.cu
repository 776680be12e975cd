// Coarse selection of long lists on tcgen05 (bf16, D = 64, top-k <= 8): gen_sparse_indices (topk.py:6-9), scores rounded to bf16.
//
// A CTA owns 128 query rows and walks the head's keys twice, 128 at a time (a job):  S = Q.K_c^T  [128 x 128] into tensor memory, thread = query row.
//   * Pass 1 keeps the maxima of 16 interleaved groups of columns per thread, 32 per row; the eighth largest bounds the row's eighth score from
//     below, and some nine scores of a row reach it, whatever its length.
//   * Pass 2 computes the same scores again and looks, eight columns at a time, for what reaches the bound.  Eight such scores are set aside in shared
//     memory as they are; they become candidates (topk_words.cuh) and go into the thread's sorted list when a warp's rows have several of them.  (Taken
//     at once, with the warp's other rows waiting, one such group cost some 500 cycles: 65 and 87 us at n = M = 4096, 8 slices, smooth and random.)
// Two warpgroups take alternate jobs (odd and even), each with two score buffers of its own, half a job each, so that the products of one half run while
// the other is looked at; they share a row's bound and merge its two lists through shared memory.  Roles: warps 0-3 / 4-7 the two groups, warp 8 TMA
// producer (queries once, a ring of two key chunks), warp 9 issues the products.
// Where there are few rows (up to 128 tiles) a cluster of two, four or eight CTAs shares a tile, each with its part of the keys.  They share their bounds
// after pass 1 and merge their lists at the end.  A score does not depend on who computes it and the candidates of a row are distinct words, so the result is the
// same for any split.  At most 256 CTAs, 32 clusters of eight: 33 and more do not run at once (n = M = 4096, 32 tiles 51 / 40 / 31 / 24 us with one, two, four and
// eight CTAs a tile, 48 tiles 56 / 47 / 36 / 44, 64 tiles 56 / 39 / 35 / 48, 96 tiles 60 / 45 / 59 / 70, 160 tiles 65 / 69).
// What bounds it: instructions of pass 2 where some row of a warp has something to set aside (nearly half of the groups of eight), two thirds of all; the
// comparisons are 64 maxima a thread and job in either pass, the tensor pipe takes 384 cycles a job.  Two CTAs share an SM, so that one's hand-overs are hidden
// by the other's work.  n = M = 4096, 8 slices: 69 us smooth, 72 random, 131 and 138 with mma.sync (topk.cu); whole layer, l1, B=2 H=4 N=65536 923 -> 856.
// The same blocks as there in all but some 2 of 100,000 rows: the sums are taken in another order.
// Every mbarrier wait is bounded.  A CTA whose wait expires computes its rows against its keys with scalar arithmetic instead (slowly, and with
// another order of the sums): a selection that went missing would not show in anything downstream.  Every CTA of a cluster comes to its meetings either way.
#include <string.h>

#include "mma_frag.cuh"
#include "tc05.cuh"
#include "tma.cuh"
#include "topk_words.cuh"

namespace llsa {

namespace {

constexpr int kRows = 128, kChunk = 128;
constexpr int kTile = kRows * 64;            // elements of a [128 x 64] bf16 tile (16 KB)
constexpr int kStages = 2;
constexpr int kThreads = 320;
constexpr int kGroups = 16;                  // column groups of a thread in pass 1
constexpr int kSlots = 12;                   // groups of eight scores that a thread sets aside in pass 2

struct CoarseMaps {
  CUtensorMap q, k;           // contiguous [BH*M, 64], [BH*n, 64], box 128 rows
};

struct CoarseBars {
  uint64_t q_full, k_full[kStages], k_empty[kStages], s_ready[4], s_free[4];      // scores: by group and half of a job
};

__device__ __forceinline__ float max3_nan(float a, float b, float c) {      // NaN if one of them is
  float d;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

__device__ __forceinline__ void store_list(void* idx_out, int idx64, int64_t at, int topk, const uint32_t (&list)[kCmTop]) {
#pragma unroll
  for (int u = 0; u < kCmTop; ++u)
    if (u < topk) {
      const uint32_t col = 65535u - (list[u] & 0xFFFFu);
      if (idx64) reinterpret_cast<int64_t*>(idx_out)[at + u] = (int64_t) col;
      else reinterpret_cast<int32_t*>(idx_out)[at + u] = (int32_t) col;
    }
}

// ---- clusters: the CTAs that share a tile of rows, each with a part of the keys
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t ld_cluster(const void* smem, uint32_t rank) {      // the word at this place of CTA `rank`'s shared memory
  uint32_t at, d;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(tc::smem_u32(smem)), "r"(rank));
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(d) : "r"(at) : "memory");
  return d;
}

// The larger half of two descending lists, descending: the larger of the ends that meet, which is a bitonic sequence
template <typename F>
__device__ __forceinline__ void list_merge(uint32_t (&list)[kCmTop], F&& other) {      // other(u): word u of the second list
  uint32_t o[kCmTop];
#pragma unroll
  for (int u = 0; u < kCmTop; ++u) o[u] = other(u);
#pragma unroll
  for (int u = 0; u < kCmTop; ++u) list[u] = umax(list[u], o[kCmTop - 1 - u]);
#pragma unroll
  for (int d = kCmTop / 2; d > 0; d >>= 1)
#pragma unroll
    for (int u = 0; u < kCmTop; ++u)
      if ((u & d) == 0) {
        const uint32_t x = umax(list[u], list[u + d]), y = umin(list[u], list[u + d]);
        list[u] = x;
        list[u + d] = y;
      }
}

// n: a multiple of 64, at most 65536.  SHARED: clusters of 1 << log_split CTAs, at most 8 and at most as many as there are chunks, share a tile of rows.
template <bool SHARED>
__global__ void __launch_bounds__(kThreads, 2)
coarse_topk_tc_kernel(const __grid_constant__ CoarseMaps maps, const bf16* __restrict__ pq, const bf16* __restrict__ pk, void* __restrict__ idx_out,
                      int idx64, int64_t M, int64_t n, int topk, int log_split, int wait_limit) {
  extern __shared__ unsigned char smem_dyn[];
  __shared__ CoarseBars bars;
  __shared__ uint32_t s_tmem;
  __shared__ tc::WaitCtl s_ctl;
  __shared__ float s_bound[SHARED ? kRows : 1];
  __shared__ int s_part[2];                              // SHARED: this CTA's first key, and how many it has
  bf16* sQ = reinterpret_cast<bf16*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));      // [128][64]
  bf16* sK = sQ + kTile;                                 // [kStages][128][64]
  // Pass 2: [slot][thread] eight scores as bf16, and their group; before and behind it the lists of maxima and of candidates, [group][row], a row's
  // words walking the banks
  uint4(*s_slot)[2 * kRows] = reinterpret_cast<uint4(*)[2 * kRows]>(sK + kStages * kTile);
  uint16_t(*s_at)[2 * kRows] = reinterpret_cast<uint16_t(*)[2 * kRows]>(s_slot + kSlots);
  uint32_t(*s_list)[kRows][kCmTop + 1] = reinterpret_cast<uint32_t(*)[kRows][kCmTop + 1]>(s_slot);
  static_assert(kSlots * 16 >= (kCmTop + 1) * 4, "room for the lists");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile tc::WaitCtl* abort_flag = &s_ctl;
  if (!SHARED) log_split = 0;
  const int rank = SHARED ? (int) blockIdx.x & ((1 << log_split) - 1) : 0;
  const int64_t bh = blockIdx.y, row0 = (int64_t) (blockIdx.x >> log_split) * kRows;
  const int chunks_all = (int) ((n + kChunk - 1) / kChunk), chunk0 = (chunks_all * rank) >> log_split;
  const int chunks = ((chunks_all * (rank + 1)) >> log_split) - chunk0, jobs = 2 * chunks;
  const volatile int* part = s_part;                     // in shared memory: a register less in the loops below
  auto key0 = [&] { return SHARED ? part[0] : 0; };
  auto keys = [&] { return SHARED ? part[1] : (int) n; };
  if (tid == 0) {
    s_part[0] = chunk0 * kChunk;
    s_part[1] = min((int) n - chunk0 * kChunk, chunks * kChunk);
    s_ctl.abort = 0;
    s_ctl.limit = wait_limit > 0 ? wait_limit : tc::kWaitPolls;
    tc::mbar_init(&bars.q_full, 1);
    for (int i = 0; i < kStages; ++i) { tc::mbar_init(&bars.k_full[i], 1); tc::mbar_init(&bars.k_empty[i], 1); }
    for (int i = 0; i < 4; ++i) { tc::mbar_init(&bars.s_ready[i], 1); tc::mbar_init(&bars.s_free[i], 4); }
    tc::fence_mbar_init();
  }
  pdl_wait();
  if (warp == 0) tc::tmem_alloc(&s_tmem, 256);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  pdl_trigger();
  const uint32_t tmem = s_tmem;

  if (SHARED && warp >= 8) cluster_arrive();                 // the bounds of pass 2 need nothing of these
  if (warp == 8) {
    // ---------------------------------------------------------------- TMA producer
    tma::expect_tx_w(&bars.q_full, kTile * 2);
    tma::load_2d_w(sQ, &maps.q, &bars.q_full, 0, (int) (bh * M + row0));      // rows past M: the next head's, or zeros; dropped
    int st = 0, c = 0;
    uint32_t ph = 1;
    for (int j = 0; j < jobs; ++j) {
      if (!tc::warp_wait(&bars.k_empty[st], ph, abort_flag)) break;
      tma::expect_tx_w(&bars.k_full[st], kTile * 2);
      tma::load_2d_w(sK + st * kTile, &maps.k, &bars.k_full[st], 0, (int) (bh * n) + key0() + c * kChunk);
      if (++st == kStages) { st = 0; ph ^= 1; }
      if (++c == chunks) c = 0;
    }
  } else if (warp == 9) {
    // ---------------------------------------------------------------- products
    const uint32_t id_s = tc::instr_desc(kRows, kChunk / 2, 0, 0);
    const uint32_t hi = (uint32_t) (tc::smem_desc(0, 0, 1024) >> 32);
    auto lo = [](const void* p) { return ((tc::smem_u32(p) >> 4) & 0x3FFFu) | ((16u >> 4) << 16); };
    constexpr uint32_t kStage = (uint32_t) (kTile * 2) >> 4;
    const uint32_t lQ = lo(sQ), lK = lo(sK);
    if (tc::warp_wait(&bars.q_full, 0, abort_flag)) {
      int st = 0;
      uint32_t ph = 0;
      for (int j = 0; j < jobs; ++j) {
        int half = 0;
        for (; half < 2; ++half) {
          const int buf = (j & 1) * 2 + half;
          // even lanes: the key chunk; odd lanes: the buffer's previous scores have been read
          const bool b = (lane & 1) && j >= 2;
          if (!tc::warp_wait(b ? &bars.s_free[buf] : &bars.k_full[st], b ? (uint32_t) ((j >> 1) - 1) & 1 : ph, abort_flag)) break;
          tc::fence_after_sync();
          tc::umma_ss_k64(tmem + buf * (kChunk / 2), lQ, hi, lK + st * kStage + half * (kStage / 2), hi, id_s);
          tc::umma_commit_w(&bars.s_ready[buf]);
        }
        if (half < 2) break;
        tc::umma_commit_w(&bars.k_empty[st]);
        if (++st == kStages) { st = 0; ph ^= 1; }
      }
    }
  } else {
    // ---------------------------------------------------------------- comparisons; thread = query row
    const int wg = warp >> 2, r = (warp & 3) * 32 + lane;
    const uint32_t t_s = tmem + ((uint32_t) ((warp & 3) * 32) << 16) + wg * kChunk;
    auto group_sync = [] { asm volatile("bar.sync 1, 256;" ::: "memory"); };
    bool ok = true;
    float v[32];
    auto ready = [&](int j, int half) {                      // half the scores of job j are there
      ok = __all_sync(0xffffffffu, tc::bounded_wait(&bars.s_ready[wg * 2 + half], (uint32_t) (j >> 1) & 1, abort_flag));
      tc::fence_after_sync();
      return ok;
    };
    auto quarter = [&](int q4) {                             // 32 columns of them
      tc::tmem_ld32_async(t_s + 32 * q4, v);
      tc::tmem_ld_wait(v);
    };
    auto give_back = [&](int half) {                         // they have been read
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tma::mbar_arrive(&bars.s_free[wg * 2 + half]);
    };
    auto halves = [&](int c) { return (c + 1) * kChunk <= keys() ? 2 : 1; };      // the last chunk may be half a chunk
    int j = wg;
    float m[kGroups];
#pragma unroll
    for (int u = 0; u < kGroups; ++u) m[u] = -CUDART_INF_F;
    for (; ok && j < chunks; j += 2) {
      const int nh = halves(j);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        if (!ready(j, half)) break;
        if (half < nh) {
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            quarter(half * 2 + q);
            if (q == 1) give_back(half);
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
              for (int e = 0; e < 8; e += 2) m[half * 8 + q * 4 + u] = fmax3(m[half * 8 + q * 4 + u], v[8 * u + e], v[8 * u + e + 1]);
          }
        } else {
          give_back(half);
        }
      }
    }
    // the eight largest of this thread's maxima, descending, then of the row's
    float best[kCmTop];
#pragma unroll
    for (int u = 0; u < kCmTop; ++u) best[u] = -CUDART_INF_F;
#pragma unroll
    for (int i = 0; i < kGroups; ++i) {
      best[kCmTop - 1] = fmaxf(best[kCmTop - 1], m[i]);
#pragma unroll
      for (int u = kCmTop - 1; u > 0; --u) {
        const float x = fmaxf(best[u - 1], best[u]), y = fminf(best[u - 1], best[u]);
        best[u - 1] = x;
        best[u] = y;
      }
    }
#pragma unroll
    for (int u = 0; u < kCmTop; ++u) s_list[wg][r][u] = __float_as_uint(best[u]);
    group_sync();
    float eighth = CUDART_INF_F;
#pragma unroll
    for (int u = 0; u < kCmTop; ++u) eighth = fminf(eighth, fmaxf(best[u], __uint_as_float(s_list[wg ^ 1][r][kCmTop - 1 - u])));
    if constexpr (SHARED) {                                  // eight scores of this CTA's keys reach that; the largest of the cluster's is the better bound
      if (wg == 0) s_bound[r] = eighth;
      __syncwarp();
      cluster_arrive();                                      // both groups have read the maxima, and the bounds are there
      cluster_wait();
#pragma unroll 1
      for (int o = 1; o < 1 << log_split; ++o) eighth = fmaxf(eighth, __uint_as_float(ld_cluster(&s_bound[r], (uint32_t) (rank ^ o))));
    } else {
      group_sync();                                          // both groups have read the maxima
    }
    uint32_t list[kCmTop], thr, w, none;
    float low;
    candidate_words(eighth, 0.f, 0u, w, none);
    bound_limits(eighth > -CUDART_INF_F ? w & 0xFFFF0000u : 0u, thr, low);      // fewer than eight groups above -inf: no bound
#pragma unroll
    for (int u = 0; u < kCmTop; ++u) list[u] = 0u;
    int held = 0;                                            // slots in use
    auto flush = [&] {                                       // what was set aside -> the list
#pragma unroll 1
      for (int u = 0; __any_sync(0xffffffffu, u < held); ++u) {
        if (u < held) {
          const uint4 x = s_slot[u][tid];
          const uint32_t p[4] = {x.x, x.y, x.z, x.w}, c = key0() + 8u * s_at[u][tid];
#pragma unroll 1
          for (int e = 0; e < 4; ++e) {
            uint32_t k[2];
            const uint32_t pe = e == 0 ? p[0] : e == 1 ? p[1] : e == 2 ? p[2] : p[3];
            candidate_words(__uint_as_float(pe << 16), __uint_as_float(pe & 0xFFFF0000u), (65535u - c - 2 * e) | ((65534u - c - 2 * e) << 16), k[0], k[1]);
#pragma unroll
            for (int i = 0; i < 2; ++i)
              if (k[i] > thr) {
                list_insert(list, k[i]);
                thr = umax(thr, list[kCmTop - 1]);
              }
          }
        }
      }
      __syncwarp();
      held = 0;
      // A full list leaves out what rounds to its last score as well: the columns that follow are larger
      if (list[kCmTop - 1]) {
        const uint32_t image = list[kCmTop - 1] >> 16, last = (image & 0x8000u ? image ^ 0x8000u : ~image & 0xFFFFu) << 16;
        low = fmaxf(low, __uint_as_float(last & 0x80000000u ? last - 1u : last + 1u));
      }
    };
    for (; ok && j < jobs; j += 2) {
      const int c = j - chunks, nq = 2 * halves(c);
#pragma unroll 1
      for (int q4 = 0; q4 < 4; ++q4) {
        if (!(q4 & 1) && !ready(j, q4 >> 1)) break;
        if (q4 < nq) quarter(q4);
        if (q4 & 1) give_back(q4 >> 1);
        if (q4 >= nq) continue;
        if (__any_sync(0xffffffffu, held > kSlots - 4)) flush();
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          float x = max3_nan(v[8 * u], v[8 * u + 1], v[8 * u + 2]);
          x = max3_nan(x, v[8 * u + 3], v[8 * u + 4]);
          x = max3_nan(x, v[8 * u + 5], v[8 * u + 6]);
          if (!(max_nan(x, v[8 * u + 7]) < low)) {           // true for NaN
            s_slot[held][tid] = make_uint4(pack_bf16(v[8 * u], v[8 * u + 1]), pack_bf16(v[8 * u + 2], v[8 * u + 3]), pack_bf16(v[8 * u + 4], v[8 * u + 5]),
                                           pack_bf16(v[8 * u + 6], v[8 * u + 7]));
            s_at[held++][tid] = (uint16_t) (c * (kChunk / 8) + q4 * 4 + u);
          }
        }
        __syncwarp();                                        // rows went different ways
      }
    }
    flush();
    group_sync();                                            // both groups are through with their slots
    if (wg == 1) {
#pragma unroll
      for (int u = 0; u < kCmTop; ++u) s_list[1][r][u] = list[u];
    }
    group_sync();
    if (wg == 0) {
      list_merge(list, [&](int u) { return s_list[1][r][u]; });
      if (SHARED) {
#pragma unroll
        for (int u = 0; u < kCmTop; ++u) s_list[0][r][u] = list[u];
      } else if (row0 + r < M && !abort_flag->abort) {
        store_list(idx_out, idx64, (bh * M + row0 + r) * topk, topk, list);
      }
    }
  }
  if (SHARED && warp >= 8) cluster_wait();
  if (abort_flag->abort) tc::abort_drain();
  tc::fence_before_sync();
  __syncthreads();
  if (abort_flag->abort && tid < kRows && row0 + tid < M) {
    const bf16* q = pq + (bh * M + row0 + tid) * 64;
    uint32_t list[kCmTop];
#pragma unroll
    for (int u = 0; u < kCmTop; ++u) list[u] = 0u;
#pragma unroll 1
    for (int c = key0(); c < key0() + keys(); ++c) {
      const bf16* k = pk + (bh * n + c) * 64;
      float acc = 0.f;
#pragma unroll 1
      for (int d = 0; d < 64; ++d) acc = fmaf(__bfloat162float(q[d]), __bfloat162float(k[d]), acc);
      uint32_t w, none;
      candidate_words(acc, 0.f, 65535u - (uint32_t) c, w, none);
      if (w > list[kCmTop - 1]) list_insert(list, w);
    }
    if (SHARED) {
#pragma unroll
      for (int u = 0; u < kCmTop; ++u) s_list[0][tid][u] = list[u];
    } else {
      store_list(idx_out, idx64, (bh * M + row0 + tid) * topk, topk, list);
    }
  }
  if constexpr (SHARED) {
    // Every CTA merges the lists of an equal share of the rows: 1 << log_split neighbouring threads read a row's list each and meet in steps.
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    if (warp < 4) {
      const int row = (kRows * rank + tid) >> log_split, others = (1 << log_split) - 1;
      uint32_t list[kCmTop];
#pragma unroll
      for (int u = 0; u < kCmTop; ++u) list[u] = ld_cluster(&s_list[0][row][u], (uint32_t) (tid & others));
#pragma unroll 1
      for (int d = 1; d <= others; d <<= 1) list_merge(list, [&](int u) { return __shfl_xor_sync(0xffffffffu, list[u], d); });
      if ((tid & others) == 0 && row0 + row < M) store_list(idx_out, idx64, (bh * M + row0 + row) * topk, topk, list);
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();                                          // nobody leaves while its lists are being read
  }
  if (warp == 0) tc::tmem_dealloc(tmem, 256);
}

}  // namespace

int launch_coarse_topk_tc(const LlsaTensor* pq, const LlsaTensor* pk, const LlsaTensor* idx, int topk, int wait_limit, cudaStream_t st) {
  const int64_t BH = pq->shape[0] * pq->shape[1], M = pq->shape[2], n = pk->shape[2];
  CoarseMaps maps;
  memset(&maps, 0, sizeof(maps));
  int rc;
  if ((rc = tma::make_map_rows(&maps.q, pq->ptr, (uint64_t) (BH * M), kRows))) return rc;
  if ((rc = tma::make_map_rows(&maps.k, pk->ptr, (uint64_t) (BH * n), kChunk))) return rc;
  const size_t smem = 1024 + (size_t) (1 + kStages) * kTile * sizeof(bf16) + (size_t) kSlots * 2 * kRows * (sizeof(uint4) + sizeof(uint16_t));
  const int64_t tiles = (M + kRows - 1) / kRows;
  int log_split = 0;                         // of how many CTAs share a tile; no influence on the result
  while (log_split < 3 && (BH * tiles) << (log_split + 1) <= 256 && n >= (int64_t) kChunk << (log_split + 1)) ++log_split;
  auto kernel = log_split ? coarse_topk_tc_kernel<true> : coarse_topk_tc_kernel<false>;
  LLSA_SMEM_LIMIT(kernel, smem);
  launch_pdl_cluster(kernel, dim3((unsigned) (tiles << log_split), (unsigned) BH), kThreads, 1u << log_split, smem, st, maps, (const bf16*) pq->ptr,
                     (const bf16*) pk->ptr, idx->ptr, idx->dtype == LLSA_I64 ? 1 : 0, M, n, topk, log_split, wait_limit);
  LLSA_LAUNCH_OK("coarse_topk_tc_kernel");
  return LLSA_OK;
}

}  // namespace llsa
