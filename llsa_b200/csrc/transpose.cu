// KV-block -> query-block index transpose used by the backward pass
// (reference: src/llsa/kernel/triton/indices_transpose.py).
//
// The reference builds the CSR with a global-atomic histogram, a cumsum and a
// second pass that claims slots with atomics, which leaves the order inside a
// bucket to chance (indices_transpose.py:23-27, :70-78).  Here it is a stable
// counting sort WITHOUT atomics: entries keep their original relative order, so
// every bucket lists its query blocks in ascending order and the output is
// bit-reproducible.
//
// transpose_range_kernel: a CTA owns a RANGE OF KEYS of one (b,h) and scans all E = M*T entries of the head twice.
//   1. the entries are cut into W contiguous segments, one per warp; a warp counts those inside the CTA's range in its own row of a
//      [W][keys of the range] table (shared-memory atomics: a count has no order).  Entries with smaller keys are counted on
//      the side: that count is the range's first position, so ranges need nothing from one another;
//   2. every key's column of the table is turned into exclusive prefixes over the segments and the column totals are scanned
//      across the range's keys -> offsets;
//   3. the warps walk their segments again, 32 entries at a time; lanes with equal keys find one another by setting their bits in the
//      key's mask word, and an entry lands at
//      offsets[key] + (count in earlier segments) + (count earlier in this segment) + (equal keys in lower lanes).
// The tables stay in shared memory whatever the number of keys, and a head occupies as many SMs as it has ranges: the scan of the
// entries is repeated per range, but they come from L2 and most lanes have nothing to do.  One CTA per head with all keys and
// __match_any_sync to group equal keys (transpose_kernel, kept for the entry point with the built-in table) took 28 us for 48 heads of
// 8,192 entries, 128 us for 5 of 40,960 and 674 us for 6 of 131,072: match.any occupies an SM for about a hundred cycles a warp (key
// ranges with it were slower still); this kernel 13, 36 and 107.
#include <mutex>

#include "common.cuh"

namespace llsa {

struct TransposeArgs {
  IdxView idx;      // [BH, M*T]
  void* offsets;    // [BH, n_kv+1]
  int off64;
  int32_t* flat;    // [BH, M*T]
  int32_t* pairs;   // [BH, M*T] or nullptr: entry position m*T + t in the order of `flat`
  int2* ranges;     // [BH, ceil(M*T / range_entries)] or nullptr: (first entry, its bucket) of the work ranges cut for the dK/dV kernel
  int range_entries;
  int64_t E;        // entries per head
  int T;
  int64_t n_kv;
  uint16_t* gtab;   // global table [BH][W][n_kv] or nullptr (shared memory)
  int32_t* status;
};

__device__ __forceinline__ int block_exclusive_scan(int v, int* warp_sums, int& block_total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) warp_sums[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int s = lane < nw ? warp_sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += t;
    }
    warp_sums[lane] = s;  // inclusive over warps
  }
  __syncthreads();
  const int before = warp > 0 ? warp_sums[warp - 1] : 0;
  block_total = warp_sums[nw - 1];
  const int excl = before + inc - v;
  __syncthreads();  // warp_sums is reused by the next call
  return excl;
}

// Work ranges of the dK/dV kernel: nominally S = range_entries entries each, but a bucket of at most S entries is never cut -- the range
// that would begin inside it begins at the bucket's first entry instead (ranges then hold 1 .. 2 S - 1 entries); only longer buckets
// are cut, at multiples of S.  The entry that lands on such a multiple knows its bucket [b0, b1).
__device__ __forceinline__ void place_range(const TransposeArgs& a, int64_t bh, int pos, int b0, int b1, int key) {
  const int S = a.range_entries;
  a.ranges[bh * (((int) a.E + S - 1) / S) + pos / S] = make_int2(b1 - b0 <= S ? b0 : pos, key);
}

// ---- one CTA per (b,h) and key range ----------------------------------------------------------------
// 32 registers a thread: 16 warps then take the room of one CTA of the dQ stage it runs beside (64 registers, as the compiler would have them, that of
// two), 32 warps that of two (62 registers: a whole SM; the limit spills 20 bytes there).  Forward + backward in us, without the limit / with it: 16 warps, two
// levels, B=3 H=5 N=5376 138.6 / 137.3, B=4 H=6 N=16384 with norms 608.9 / 606.4, one level, B=4 H=6 N=4096 175.3 / 176.1; 32 warps, B=1 H=5 N=40960 top-16
// 499.7 / 493.9 (in a graph 489.3 / 491.8), B=1 H=6 N=65536 601.0 / 602.6; alone on its stream, fp32, B=1 H=2 N=1024, 96.3 / 96.4.
template <int W>
__global__ void __launch_bounds__(W * 32, 64 / W) transpose_range_kernel(TransposeArgs a, int keys_per_range, uint32_t t_magic) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ int warp_sums[32];
  __shared__ int s_below[W], s_kept[W];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t bh = blockIdx.x;                         // any number of heads: the x axis has no 65,535 limit
  const int E = (int) a.E, n = (int) a.n_kv, lo = (int) blockIdx.y * keys_per_range, K = min(keys_per_range, n - lo);
  const bool last = (int) blockIdx.y + 1 == (int) gridDim.y;
  int* base = reinterpret_cast<int*>(smraw);             // [K + 1]
  int* tab = base + keys_per_range + 1;                  // [W][K] entries seen, then [W][K] lanes that hold the key right now
  for (int i = threadIdx.x; i < 2 * W * K; i += blockDim.x) tab[i] = 0;
  __syncthreads();

  const int L = ((E + W - 1) / W + 31) / 32 * 32, seg0 = min(E, warp * L), seg1 = min(E, seg0 + L);
  const int64_t* idx64 = reinterpret_cast<const int64_t*>(a.idx.p) + bh * E;
  const int32_t* idx32 = reinterpret_cast<const int32_t*>(a.idx.p) + bh * E;
  int32_t* flat = a.flat + bh * E;
  int32_t* pairs = a.pairs ? a.pairs + bh * E : nullptr;
  // a key outside [0, n) (whatever its upper half holds) comes back as -1
  auto key_at = [&](int e) -> int {
    if (!a.idx.is64) return idx32[e];
    const int64_t k = idx64[e];
    return k < 0 || k >= n ? -1 : (int) k;
  };
  int* mytab = tab + warp * K;
  unsigned* mymask = reinterpret_cast<unsigned*>(tab + (W + warp) * K);
  const unsigned lt_mask = (1u << lane) - 1u;
  // walk(f): f(entry, key - lo, inside the range) for 32 entries at a time, four loads ahead
  auto walk = [&](auto&& f) {
    constexpr int AHEAD = 4;
    int key[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const int e = seg0 + u * 32 + lane;
      key[u] = e < seg1 ? key_at(e) : -1;
    }
    for (int e0 = seg0; e0 < seg1; e0 += 32 * AHEAD) {
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        const int e = e0 + u * 32 + lane, en = e + 32 * AHEAD, k = key[u];
        key[u] = en < seg1 ? key_at(en) : -1;
        f(e, k, e < seg1);
      }
    }
  };

  // ---- 1: per-segment histograms of the range, entries below it
  int below = 0, kept = 0;
  walk([&](int e, int k, bool real) {
    const bool valid = real && k >= 0 && k < n;
    if (real && !valid && last && a.status) atomicOr(a.status, (int) LLSA_DEV_BAD_INDEX);
    below += valid && k < lo;
    kept += valid;
    const int kk = k - lo;
    if (valid && kk >= 0 && kk < K) atomicAdd(&mytab[kk], 1);
  });
  below = __reduce_add_sync(0xffffffffu, below);
  kept = __reduce_add_sync(0xffffffffu, kept);
  if (lane == 0) { s_below[warp] = below; s_kept[warp] = kept; }
  __syncthreads();
  int total_entries = 0, carry = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) { carry += s_below[w]; total_entries += s_kept[w]; }

  // ---- 2: per-key prefix over segments, then scan of the totals over the range's keys
  for (int j0 = 0; j0 < K; j0 += blockDim.x) {
    const int j = j0 + threadIdx.x;
    int run = 0;
    if (j < K) {
#pragma unroll
      for (int s = 0; s < W; ++s) {
        const int c = tab[s * K + j];
        tab[s * K + j] = run;
        run += c;
      }
    }
    int total;
    const int excl = block_exclusive_scan(run, warp_sums, total);
    if (j < K) {
      base[j] = carry + excl;
      if (a.off64) reinterpret_cast<int64_t*>(a.offsets)[bh * (n + 1) + lo + j] = carry + excl;
      else reinterpret_cast<int32_t*>(a.offsets)[bh * (n + 1) + lo + j] = carry + excl;
    }
    carry += total;
  }
  if (threadIdx.x == 0) {
    base[K] = carry;
    if (last) {
      if (a.off64) reinterpret_cast<int64_t*>(a.offsets)[bh * (n + 1) + n] = carry;
      else reinterpret_cast<int32_t*>(a.offsets)[bh * (n + 1) + n] = carry;
    }
  }
  __syncthreads();
  // work ranges that lie wholly behind the last entry (entries were dropped, or E is not a multiple of the range size) are empty
  if (a.ranges && last) {
    const int R = (E + a.range_entries - 1) / a.range_entries;
    for (int r = total_entries / a.range_entries + threadIdx.x; r < R; r += blockDim.x)
      if (r * a.range_entries >= total_entries) a.ranges[bh * R + r] = make_int2(total_entries, n - 1);
  }

  // ---- 3: stable fill
  walk([&](int e, int k, bool real) {
    const int kk = k - lo;
    const bool in = real && k >= 0 && k < n && kk >= 0 && kk < K;
    if (!__any_sync(0xffffffffu, in)) return;
    if (in) atomicOr(&mymask[kk], 1u << lane);
    __syncwarp();
    unsigned peers = 0;
    int seen = 0;
    if (in) {
      peers = mymask[kk];
      seen = mytab[kk];
      const int pos = base[kk] + seen + __popc(peers & lt_mask);
      int m = t_magic == 0u ? e : (int) __umulhi((uint32_t) e, t_magic);      // e / T, or one more where e * T passes 2^32
      m -= (int64_t) m * a.T > e;
      flat[pos] = m;
      if (pairs) pairs[pos] = e;
      if (a.ranges && (pos & (a.range_entries - 1)) == 0) place_range(a, bh, pos, base[kk], base[kk + 1], k);
    }
    __syncwarp();
    if (in && (peers & lt_mask) == 0) {
      mytab[kk] = seen + __popc(peers);
      mymask[kk] = 0u;
    }
    __syncwarp();
  });
}

// ---- one CTA per (b,h), all keys, the count table in shared or global memory ------------------------
__global__ void __launch_bounds__(1024) transpose_kernel(TransposeArgs a) {
  extern __shared__ unsigned char smraw[];
  __shared__ int warp_sums[32];
  const int W = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t bh = blockIdx.x, n = a.n_kv, E = a.E;
  int* base = reinterpret_cast<int*>(smraw);                                        // [n_kv]
  uint16_t* tab = a.gtab ? a.gtab + bh * W * n : reinterpret_cast<uint16_t*>(base + n);  // [W][n_kv]

  for (int64_t i = threadIdx.x; i < (int64_t) W * n; i += blockDim.x) tab[i] = 0;
  __syncthreads();

  int64_t L = (E + W - 1) / W;
  L = (L + 31) / 32 * 32;
  const int64_t seg0 = min(E, warp * L), seg1 = min(E, seg0 + L);
  uint16_t* mytab = tab + (int64_t) warp * n;
  const unsigned lt_mask = (1u << lane) - 1u;

  // ---- 1: per-segment histograms
  for (int64_t e0 = seg0; e0 < seg1; e0 += 32) {
    const int64_t e = e0 + lane;
    bool valid = e < seg1;
    int64_t key = valid ? a.idx.at(bh * E + e) : -1;
    if (valid && (key < 0 || key >= n)) {
      if (a.status) atomicOr(a.status, (int) LLSA_DEV_BAD_INDEX);
      valid = false;
    }
    const unsigned act = __ballot_sync(0xffffffffu, valid);
    if (valid) {
      const unsigned peers = __match_any_sync(act, (int) key);
      if ((peers & lt_mask) == 0) mytab[key] = (uint16_t) (mytab[key] + __popc(peers));
    }
    __syncwarp();
  }
  __syncthreads();

  // ---- 2: per-key prefix over segments, then scan of the totals over keys
  int carry = 0;
  for (int64_t j0 = 0; j0 < n; j0 += blockDim.x) {
    const int64_t j = j0 + threadIdx.x;
    int run = 0;
    if (j < n) {
      for (int s = 0; s < W; ++s) {
        const int c = tab[(int64_t) s * n + j];
        tab[(int64_t) s * n + j] = (uint16_t) run;
        run += c;
      }
      // the prefixes are 16-bit: a key listed more than 65535 times in one head (possible only when rows repeat a key)
      // cannot be placed; the fill below then skips what would fall outside and the status word says so
      if (run > 65535 && a.status) atomicOr(a.status, (int) LLSA_DEV_BAD_INDEX);
    }
    int total;
    const int excl = block_exclusive_scan(run, warp_sums, total);
    if (j < n) {
      base[j] = carry + excl;
      if (a.off64) reinterpret_cast<int64_t*>(a.offsets)[bh * (n + 1) + j] = carry + excl;
      else reinterpret_cast<int32_t*>(a.offsets)[bh * (n + 1) + j] = carry + excl;
    }
    carry += total;
  }
  if (threadIdx.x == 0) {
    if (a.off64) reinterpret_cast<int64_t*>(a.offsets)[bh * (n + 1) + n] = carry;
    else reinterpret_cast<int32_t*>(a.offsets)[bh * (n + 1) + n] = carry;
  }
  __syncthreads();
  // ---- 3: stable fill
  for (int64_t e0 = seg0; e0 < seg1; e0 += 32) {
    const int64_t e = e0 + lane;
    bool valid = e < seg1;
    int64_t key = valid ? a.idx.at(bh * E + e) : -1;
    if (valid && (key < 0 || key >= n)) valid = false;
    const unsigned act = __ballot_sync(0xffffffffu, valid);
    unsigned peers = 0;
    int seen = 0;
    if (valid) {
      peers = __match_any_sync(act, (int) key);
      seen = mytab[key];
      const int pos = base[key] + seen + __popc(peers & lt_mask);
      if (pos < E) {
        a.flat[bh * E + pos] = (int32_t) (e / a.T);
      }
    }
    __syncwarp();
    if (valid && (peers & lt_mask) == 0) mytab[key] = (uint16_t) (seen + __popc(peers));
    __syncwarp();
  }
}

// Chooses the warp count W and where the [W][n_kv] count table lives.  Returns
// W (8, 16 or 32); *global is set when the table does not fit in shared memory
// or the segments would overflow the 16-bit counters with fewer warps.
static int plan_transpose(int64_t n_kv, int64_t E, size_t* smem, bool* global) {
  const size_t limit = 200 * 1024;
  for (int W = 32; W >= 8; W >>= 1) {
    const size_t need = (size_t) n_kv * 4 + (size_t) W * n_kv * 2;
    if (need <= limit && (E + W - 1) / W + 32 <= 65535) {
      *smem = need;
      *global = false;
      return W;
    }
  }
  *smem = (size_t) n_kv * 4;
  *global = true;
  return 32;
}

}  // namespace llsa

using namespace llsa;

extern "C" int llsa_transpose_range_entries(int64_t B, int64_t H, int64_t M, int64_t T) {
  // The size also picks the dK/dV kernel's form (attn_bwd_mma.cu): spans, one per warp, for ranges of 16, windows for ranges of 32.  Forward + backward
  // in a graph, us, spans / windows: one level, N = 16384: 2,048 ranges (of 32) 311 / 320, 3,072 464 / 458, 4,096 590 / 604, 4,608 690 / 691, N = 4096:
  // 4,608 402 / 399; two levels, N = 16384: 3,072 268 / 271, 3,840 322 / 324, 4,608 385 / 382, N = 40960: 3,200 338 / 343, 3,840 397 / 402, N = 65536:
  // 4,096 403 / 419.  Above, spans fall behind (6,144 ranges 642 / 616, 6,400 547 / 536): warps far apart in the list no longer meet in L2.
  const int64_t ranges = B * H * ((M * T + kRangeEntries - 1) / kRangeEntries);
  return ranges < 2 * 148 * 8 * 2 ? kRangeEntriesSmall : kRangeEntries;
}

extern "C" size_t llsa_transpose_scratch_bytes(int64_t B, int64_t H, int64_t M, int64_t T, int64_t n_kv) {
  size_t smem;
  bool global;
  plan_transpose(n_kv, M * T, &smem, &global);
  return global ? (size_t) B * H * 32 * n_kv * 2 : 0;
}

static int transpose_impl(const LlsaTensor* idx, const LlsaTensor* offsets, const LlsaTensor* flat, const LlsaTensor* pairs,
                          const LlsaTensor* ranges, int64_t n_kv, int32_t* status, void* stream) {
  LLSA_REQUIRE(idx && offsets && flat && idx->ptr && offsets->ptr && flat->ptr, LLSA_ERR_NULL, "transpose_indices: null tensor");
  LLSA_REQUIRE(idx->ndim == 4, LLSA_ERR_SHAPE, "transpose_indices: idx must be [B,H,M,T]");
  const int64_t B = idx->shape[0], H = idx->shape[1], M = idx->shape[2], T = idx->shape[3];
  LLSA_REQUIRE(is_index_dtype(idx->dtype) && is_index_dtype(offsets->dtype) && flat->dtype == LLSA_I32, LLSA_ERR_DTYPE,
               "transpose_indices: idx/offsets must be i32 or i64, flat i32");
  LLSA_REQUIRE(n_kv >= 1 && n_kv < (1ll << 31) && T >= 1, LLSA_ERR_ARG, "transpose_indices: bad n_kv=%lld", (long long) n_kv);
  const int64_t E = M * T;
  LLSA_REQUIRE(E <= 32ll * 65504, LLSA_ERR_SHAPE, "transpose_indices: M*T=%lld exceeds the supported %lld", (long long) E, 32ll * 65504);
  const int64_t si[4] = {B, H, M, T}, so[3] = {B, H, n_kv + 1}, sf[3] = {B, H, E};
  int rc;
  if ((rc = check_contig(idx, "idx", idx->dtype, 4, si))) return rc;
  if ((rc = check_contig(offsets, "offsets", offsets->dtype, 3, so))) return rc;
  if ((rc = check_contig(flat, "flat", LLSA_I32, 3, sf))) return rc;
  if (pairs && (rc = check_contig(pairs, "pairs", LLSA_I32, 3, sf))) return rc;
  int S = kRangeEntries;
  if (ranges) {
    LLSA_REQUIRE(ranges->ndim == 4, LLSA_ERR_SHAPE, "transpose_indices_pairs: ranges must be [B,H,R,2]");
    S = range_entries_of(E, ranges->shape[2]);
    LLSA_REQUIRE(S > 0, LLSA_ERR_SHAPE, "transpose_indices_pairs: ranges holds %lld ranges; expected ceil(%lld / %d) or ceil(%lld / %d)",
                 (long long) ranges->shape[2], (long long) E, kRangeEntries, (long long) E, kRangeEntriesSmall);
    const int64_t sr[4] = {B, H, (E + S - 1) / S, 2};
    if ((rc = check_contig(ranges, "ranges", LLSA_I32, 4, sr))) return rc;
  }
  // the per-key prefixes over the segments are 16-bit: with distinct keys inside a row a key occurs at most M times per head
  LLSA_REQUIRE(M <= 65535, LLSA_ERR_SHAPE, "transpose_indices: M=%lld query blocks per head exceed the supported 65535", (long long) M);
  LLSA_REQUIRE((int64_t) n_kv * 4 <= 200 * 1024, LLSA_ERR_SHAPE, "transpose_indices: n_kv=%lld too large", (long long) n_kv);
  if (B * H == 0) return LLSA_OK;
  TransposeArgs a;
  a.idx = make_idx(idx);
  a.offsets = offsets->ptr;
  a.off64 = offsets->dtype == LLSA_I64;
  a.flat = (int32_t*) flat->ptr;
  a.pairs = pairs ? (int32_t*) pairs->ptr : nullptr;
  a.ranges = ranges ? (int2*) ranges->ptr : nullptr;
  a.range_entries = S;
  a.E = E;
  a.T = (int) T;
  a.n_kv = n_kv;
  a.gtab = nullptr;
  a.status = status;
  // e / T from the high half of e * ceil(2^32 / T); T = 1 is marked by 0
  const uint32_t t_magic = T == 1 ? 0u : (uint32_t) (((1ull << 32) + T - 1) / (uint64_t) T);
  // Warps: a warp's walk is a chain of some 300 cycles per 32 entries, so long lists get 32 (5 heads of 40,960 entries: 36 us against 46
  // with 16), short ones 16 (fewer rows to clear and to scan: 24 heads of 2,048 entries 5.5 us against 6.9).  Ranges: about 96 CTAs on the
  // GPU, since every range scans the whole list (48 heads of 8,192 entries: 13 us with 2 ranges, 19 with 4), at least 128 keys each,
  // the tables within shared memory.
  const int warps = E > 16384 ? 32 : 16;
  const int64_t most_keys = (196 * 1024 / 4 - 1) / (2 * warps + 1);
  int64_t ranges_per_head = (96 + B * H - 1) / (B * H);
  const int64_t most = (n_kv + 127) / 128, fewest = (n_kv + most_keys - 1) / most_keys;
  ranges_per_head = ranges_per_head > most ? most : ranges_per_head;
  ranges_per_head = ranges_per_head < fewest ? fewest : ranges_per_head;
  const int keys = (int) ((n_kv + ranges_per_head - 1) / ranges_per_head);
  const dim3 grid((unsigned) (B * H), (unsigned) ((n_kv + keys - 1) / keys));
  const size_t smem = ((size_t) keys * (2 * warps + 1) + 1) * sizeof(int);
  cudaStream_t st = (cudaStream_t) stream;
  if (warps == 32) {
    LLSA_SMEM_LIMIT((transpose_range_kernel<32>), smem);
    launch_pdl(transpose_range_kernel<32>, grid, 32 * 32, smem, st, a, keys, t_magic);
  } else {
    LLSA_SMEM_LIMIT((transpose_range_kernel<16>), smem);
    launch_pdl(transpose_range_kernel<16>, grid, 16 * 32, smem, st, a, keys, t_magic);
  }
  LLSA_LAUNCH_OK("transpose_range_kernel");
  return LLSA_OK;
}

extern "C" int llsa_transpose_indices(const LlsaTensor* idx, const LlsaTensor* offsets, const LlsaTensor* flat, int64_t n_kv,
                                      void* scratch, size_t scratch_bytes, int32_t* status, void* stream) {
  if (idx && idx->ndim == 4 && n_kv >= 1) {      // what this entry point asks for by contract, although no table lives there any more
    const size_t need = llsa_transpose_scratch_bytes(idx->shape[0], idx->shape[1], idx->shape[2], idx->shape[3], n_kv);
    LLSA_REQUIRE(need == 0 || (scratch && scratch_bytes >= need), LLSA_ERR_WORKSPACE, "transpose_indices: needs %zu bytes of scratch", need);
  }
  return transpose_impl(idx, offsets, flat, nullptr, nullptr, n_kv, status, stream);
}

extern "C" int llsa_transpose_indices_pairs(const LlsaTensor* idx, const LlsaTensor* offsets, const LlsaTensor* flat, const LlsaTensor* pairs,
                                            const LlsaTensor* ranges, int64_t n_kv, void* scratch, size_t scratch_bytes, int32_t* status,
                                            void* stream) {
  (void) scratch;
  (void) scratch_bytes;
  return transpose_impl(idx, offsets, flat, pairs, ranges, n_kv, status, stream);
}

// ---------------------------------------------------------------------------
// llsa_transpose_indices_noalloc: the same index transpose for callers that
// cannot hand over a scratch buffer.
//
// Some hosts of this library never get to call cudaMalloc themselves: a
// serving or training process that gave the whole device to its own memory
// arena at start-up, or a plugin runtime that only passes input and output
// buffers across its boundary.  For the long-sequence shapes (n_kv above a few
// thousand KV blocks) llsa_transpose_indices needs B*H*32*n_kv*2 bytes of
// device scratch for its count table; here that table lives in a fixed array
// inside the library image instead.  Every GPU that loads the library carries
// the array (kNoAllocScratchBytes) until the process exits.
//
// The array's name is only a host-side handle: its device address is looked up
// once per device with cudaGetSymbolAddress (with that device current) and the
// address -- not the symbol -- is what the kernel receives.
namespace llsa {

constexpr size_t kNoAllocScratchBytes = 8u << 20;   // 8 MiB: e.g. B*H = 6 heads of 262144 tokens (n_kv = 16384)
static __device__ __align__(256) unsigned char g_transpose_scratch[kNoAllocScratchBytes];

constexpr int kMaxDevices = 64;
static void* g_scratch_addr[kMaxDevices];   // device address of g_transpose_scratch, per device ordinal
static bool g_scratch_ready[kMaxDevices];
static std::mutex g_scratch_mutex;

// Device address of the static scratch on the CURRENT device (looked up on first use there).
static int noalloc_scratch(void** out) {
  int dev = -1;
  LLSA_CUDA_OK(cudaGetDevice(&dev));
  LLSA_REQUIRE(dev >= 0 && dev < kMaxDevices, LLSA_ERR_ARG, "transpose_indices_noalloc: device ordinal %d unsupported", dev);
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (!g_scratch_ready[dev]) {
    void* p = nullptr;
    LLSA_CUDA_OK(cudaGetSymbolAddress(&p, g_transpose_scratch));
    LLSA_REQUIRE(p != nullptr, LLSA_ERR_CUDA, "transpose_indices_noalloc: no device address for the static scratch");
    g_scratch_addr[dev] = p;
    g_scratch_ready[dev] = true;
  }
  *out = g_scratch_addr[dev];
  return LLSA_OK;
}

}  // namespace llsa

extern "C" int llsa_transpose_indices_noalloc(const LlsaTensor* idx, const LlsaTensor* offsets, const LlsaTensor* flat, int64_t n_kv,
                                              int32_t* status, void* stream) {
  LLSA_REQUIRE(idx && offsets && flat && idx->ptr && offsets->ptr && flat->ptr, LLSA_ERR_NULL, "transpose_indices_noalloc: null tensor");
  LLSA_REQUIRE(idx->ndim == 4, LLSA_ERR_SHAPE, "transpose_indices_noalloc: idx must be [B,H,M,T]");
  const int64_t B = idx->shape[0], H = idx->shape[1], M = idx->shape[2], T = idx->shape[3];
  LLSA_REQUIRE(is_index_dtype(idx->dtype) && is_index_dtype(offsets->dtype) && flat->dtype == LLSA_I32, LLSA_ERR_DTYPE,
               "transpose_indices_noalloc: idx/offsets must be i32 or i64, flat i32");
  LLSA_REQUIRE(n_kv >= 1 && n_kv < (1ll << 31) && T >= 1, LLSA_ERR_ARG, "transpose_indices_noalloc: bad n_kv=%lld", (long long) n_kv);
  const int64_t E = M * T;
  LLSA_REQUIRE(E <= 32ll * 65504, LLSA_ERR_SHAPE, "transpose_indices_noalloc: M*T=%lld exceeds the supported %lld", (long long) E,
               32ll * 65504);
  const int64_t si[4] = {B, H, M, T}, so[3] = {B, H, n_kv + 1}, sf[3] = {B, H, E};
  int rc;
  if ((rc = check_contig(idx, "idx", idx->dtype, 4, si))) return rc;
  if ((rc = check_contig(offsets, "offsets", offsets->dtype, 3, so))) return rc;
  if ((rc = check_contig(flat, "flat", LLSA_I32, 3, sf))) return rc;
  // the count table [B*H][32 warps][n_kv] of 16-bit counters always goes to the static array
  const size_t need = (size_t) B * H * 32 * (size_t) n_kv * 2;
  LLSA_REQUIRE(need <= kNoAllocScratchBytes, LLSA_ERR_WORKSPACE,
               "transpose_indices_noalloc: B*H*n_kv = %lld needs %zu bytes of count table, the built-in scratch holds %zu "
               "(use llsa_transpose_indices with caller scratch)", (long long) (B * H * n_kv), need, (size_t) kNoAllocScratchBytes);
  const size_t smem = (size_t) n_kv * 4;   // per-key bases stay in shared memory
  LLSA_REQUIRE(smem <= 200 * 1024, LLSA_ERR_SHAPE, "transpose_indices_noalloc: n_kv=%lld too large", (long long) n_kv);
  LLSA_REQUIRE(M <= 65535, LLSA_ERR_SHAPE, "transpose_indices_noalloc: M=%lld query blocks per head exceed the supported 65535", (long long) M);
  if (B * H == 0) return LLSA_OK;
  void* tab = nullptr;
  if ((rc = noalloc_scratch(&tab))) return rc;
  TransposeArgs a;
  a.idx = make_idx(idx);
  a.offsets = offsets->ptr;
  a.off64 = offsets->dtype == LLSA_I64;
  a.flat = (int32_t*) flat->ptr;
  a.E = E;
  a.T = (int) T;
  a.n_kv = n_kv;
  a.gtab = (uint16_t*) tab;     // the kernel zero-fills the part of the table it uses before counting
  a.status = status;
  LLSA_SMEM_LIMIT((transpose_kernel), smem);
  transpose_kernel<<<(unsigned) (B * H), 32 * 32, smem, (cudaStream_t) stream>>>(a);
  LLSA_LAUNCH_OK("transpose_kernel");
  return LLSA_OK;
}
