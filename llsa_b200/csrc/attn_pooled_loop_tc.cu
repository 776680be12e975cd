// Pooled stages of the LLSA forward on tcgen05 for LONG pooled key lists: a key loop over 128-key chunks.
//
// attn_pooled_tc.cu keeps all pooled keys of a tile in tensor memory at once and therefore stops at 192 keys.
// Here a tile of 128 query rows walks its pooled keys chunk by chunk:
//   one level  (sparse_attention_res_1.py:85-106): ALL N/16 level-1 pooled keys, weight token_weight;
//   two levels (sparse_attention_res_2.py:94-149): first the level-1 children of the parent's selected level-2 blocks (gathered,
//              eight blocks to a chunk, weight token_weight), then ALL N/256 level-2 keys (weight token_weight_2).
// Both lists may end inside a chunk (at a multiple of 32 keys): what lies behind the end is loaded (a repeated block, or the rows
// that follow in memory) and neither exponentiated nor multiplied: the softmax warps and the P.V steps stop at the list's end.
// Two passes over the chunks make the softmax exact without rescaling an accumulator that lives in TMEM:
//   pass 1: S = Q.K_c^T per chunk, row maxima only;
//   pass 2: S again, P = exp2(S*scale*log2e + log2 w - max) written back into TMEM over S (packed bf16) and used as
//           the A operand of O += P.V_c; row sums on the side.
// With a `redo` byte per query row from the caller the first pass is dropped: the pooled part only ever meets the fine
// part through their log-sum-exp, so the fine part's log-sum-exp (already known per row) serves as the reference of the
// exponentials, P = exp2(S' - lse_fine) (REM: moved up to a quarter above a power of two, kRefShift).  Anything below 2^-126 of the fine part's weight is irrelevant, and bf16 / fp32
// hold anything up to 2^127 times it; a row whose pooled keys outweigh its fine keys by more than that (its row sum
// passes 1e30, or is NaN) is left untouched and marked in `redo`; a CTA that has marked a row of its tiles goes over them again
// with two passes and writes exactly the marked rows.  (A second launch that looked for marks cost every call 1 to 2 us.)
// Roles (one persistent CTA per SM, 16 or 20 warps; warps 8 to 11 run in step, tc05.cuh: umma_ss_k64):
//   warp 8, warp 11  : TMA producers: Q per tile (2 stages) and K chunks (ring of 4; every chunk is loaded in both passes); V chunks (ring
//                      of 4, pass 2 only)
//   warp 9           : issues S of every "job" (a chunk of a pass).  Job number n, counted over all tiles of the CTA,
//                      uses S buffer n mod 3 (TMEM columns [128 b, 128 b + 128)); O of tile i lives in [384 + 64 (i mod 2), + 64).
//   warp 10          : issues O += P.V of the pass-2 jobs and hands every job's buffer back to warp 9 (buf_free,
//                      committed behind the instructions that read P)
//   warps 0-3 / 4-7 (/ 16-19) : two or three softmax warpgroups (GROUPS), group w owns the jobs n = w (mod GROUPS); thread r owns query row r (TMEM
//                      lane r).  They leave a row's sum (and reference) in shared memory and go on to the next tile.
//   warps 12-15      : epilogue, thread = row: merges O with the fine part (o, lse written by the fine kernel) and stores both.
// What bounds it: the chain S -> exponentials -> P.V over three buffers, 1,430 cycles a job: with the softmax left out the copies, products and
// hand-overs of a job take 900, with its exponentials alone left out 1,090; the 128 exponentials of a row take 1,024 on the SM's 16 MUFU lanes.
// Two groups' warps spend two thirds of a job in waits and loads; a third one takes turns with them where tiles are long enough (kThreeGroupKeys):
// l1, B=2 H=4 N=65536: 692 us with two, 669 with three; two levels, H=6 N=262144: 620 -> 590; B=2 H=4 N=65536: 90 -> 85.  No gain from: two
// groups that load a whole row of scores at once and hand the S buffer back before the exponentials (732: fewer warps for the MUFU); a quarter
// or a third of the exponentials as a degree-5 polynomial on the FMA pipe (669 and 676; 85 -> 95 and 98 at N=65536 two levels).  Eight warps a job
// were 2 % faster on long lists (657) and 4 % slower on short ones (56 -> 58).  In the form with one producer lane, the epilogue in the softmax
// groups and one O buffer (785 us) the producer needed 1,300 cycles a job for its two waits and two copies, and every tile boundary cost 5,900
// idle cycles.
// Every mbarrier wait is bounded; a wait that expires raises a CTA-wide abort flag, every role leaves its loops, the epilogue puts NaN into lse of
// every row of the CTA (poison_lse) and TMEM is freed.
#include <string.h>

#include "attn.cuh"
#include "mma_frag.cuh"
#include "tc05.cuh"
#include "tma.cuh"

namespace llsa {

namespace {

constexpr int kRows = 128;
constexpr int kChunk = 128;                 // keys per chunk
constexpr int kTile = kRows * 64;           // elements of a [128 x 64] bf16 tile (16 KB)
constexpr int kKStages = 4, kVStages = 4;
constexpr int kBufs = 3;                    // S buffers
// Registers of a thread, per role.  Three softmax groups share what 640 threads launch with: 40 + 104 + 3 x 112 = 5 x 96; with two every thread keeps
// the 128 of the launch.
template <int GROUPS>
struct Split {
  static constexpr int kThreads = GROUPS == 3 ? 640 : 512, kLaunch = GROUPS == 3 ? 96 : 128;
  static constexpr int kIssue = GROUPS == 3 ? 40 : kLaunch, kEpilogue = GROUPS == 3 ? 104 : kLaunch, kSoftmax = GROUPS == 3 ? 112 : kLaunch;
  static_assert(kIssue + kEpilogue + GROUPS * kSoftmax <= (2 + GROUPS) * kLaunch, "the takers would wait for good");
};
constexpr float kLog2eF = 1.4426950408889634f;
constexpr uint32_t kColO = 384;
// One pass over a list that one kernel used to take with running maxima (REM): where in its binade a probability of a logit of 0 lands.  bf16 is finest just below a power of two, which is where a row's
// maximum as reference puts the largest ones; a reference at no particular place costs up to 12 % of o's error where the keys weigh about alike
// (against fp64, N(0,1) inputs, two levels, N = 40960, top-16: 2.33e-3; 2.33e-3, 2.11e-3, 2.10e-3, 2.15e-3, 2.22e-3 with the reference at
// 0, 1/8, 1/4, 3/8, 1/2 above a power of two; 2.09e-3 with two passes, 2.07e-3 in one kernel).  The weights 16 and 256 are powers of two.
constexpr float kRefShift = 0.25f;

// Pooled keys of a row from which three softmax groups are the better split; below, a tile is a few jobs, and every group of it costs the tile a
// round of hand-overs (sums, maxima, the next tile's reference).  Lists whose fine part comes with a remainder gain later: their epilogue is longer.
// Whole forward in us, two groups / three: one level, B=2 H=6, 256 keys 30.9 / 31.5, 512 57.5 / 56.5, 608 (remainder) 126.6 / 125.1; two levels, B=3
// H=6 N=32768, 256 keys 238 / 242; H=6 N=24576, 256 (160 + 96) 93 / 96, remainder; H=6 N=16384, 320 and 384, remainder, 69 / 70 and 99 / 100; H=6
// N=65536, 384 keys 178 / 174, 448 with remainder 254 / 263; H=5 N=40960, 480 with remainder 184.5 / 184.1.
constexpr int kThreeGroupKeys = 384, kThreeGroupKeysRem = 480;

struct LoopMaps {
  CUtensorMap q;              // [B,H,Nq,64] 4-D, box 128 rows
  CUtensorMap kg, vg;         // gathered level-1 keys / values (two levels): [BH*n1, 64], box 16 rows
  CUtensorMap kc, vc;         // contiguous pooled keys / values: [BH*n, 64], box 128 rows
};

struct LoopBars {
  uint64_t q_full[2], q_empty[2], k_full[kKStages], k_empty[kKStages], v_full[kVStages], v_empty[kVStages];
  uint64_t s_ready[kBufs], wg_done[kBufs], buf_free[kBufs], o_ready[2], o_free[2], sum_ready[2], xchg;
};

template <int GROUPS>
__device__ __forceinline__ void init_bars(LoopBars& bars) {
  for (int i = 0; i < 2; ++i) {
    tc::mbar_init(&bars.q_full[i], 1);
    tc::mbar_init(&bars.q_empty[i], 1);
  }
  for (int i = 0; i < kBufs; ++i) {
    tc::mbar_init(&bars.s_ready[i], 1);
    tc::mbar_init(&bars.wg_done[i], 4);         // one arrival per warp of the group
    tc::mbar_init(&bars.buf_free[i], 1);
  }
  for (int i = 0; i < kKStages; ++i) { tc::mbar_init(&bars.k_full[i], 1); tc::mbar_init(&bars.k_empty[i], 1); }
  for (int i = 0; i < kVStages; ++i) { tc::mbar_init(&bars.v_full[i], 1); tc::mbar_init(&bars.v_empty[i], 1); }
  for (int i = 0; i < 2; ++i) {
    tc::mbar_init(&bars.o_ready[i], 1);
    tc::mbar_init(&bars.o_free[i], 4);
    tc::mbar_init(&bars.sum_ready[i], 4 * GROUPS);
  }
  tc::mbar_init(&bars.xchg, 4 * GROUPS);
  tc::fence_mbar_init();
}

// n_chunks: chunks per tile; gathered: how many of them, the first ones, are gathered level-1 blocks (two levels); n_c: rows per
// head of the contiguous pooled tensor.  REM: the fine part of o is the bf16 value in o plus its remainder in a.rem; AHEAD: the launch.
template <bool REM, int GROUPS, bool AHEAD = false>
__global__ void __launch_bounds__(Split<GROUPS>::kThreads, 1)
attn_fwd_pooled_loop_tc_kernel(AttnP<bf16> a, const __grid_constant__ LoopMaps maps, int n_chunks, int gathered, int64_t n_c, int n_tiles,
                               int tiles_per_head, unsigned char* redo) {
  extern __shared__ unsigned char smem_dyn[];
  __shared__ LoopBars bars_of[2];                    // of the first round over the tiles and of the one for marked rows
  __shared__ uint32_t s_tmem;
  __shared__ tc::WaitCtl s_ctl;
  __shared__ float s_max[2][GROUPS][kRows];             // [tile parity][group][row]: row maxima after pass 1
  __shared__ float s_sum[2][GROUPS][kRows], s_ref[2][kRows];      // [tile parity][group][row] row sums; [tile parity][row] their reference
  bf16* base = reinterpret_cast<bf16*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  bf16* sQ = base;                          // [2][128][64]
  bf16* sK = sQ + 2 * kTile;                // [kKStages][128][64]
  bf16* sV = sK + kKStages * kTile;         // [kVStages][128][64]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile tc::WaitCtl* abort_flag = &s_ctl;
  const int n_my = (n_tiles - (int) blockIdx.x + (int) gridDim.x - 1) / (int) gridDim.x;
  if (tid == 0) {
    s_ctl.abort = 0;
    s_ctl.limit = a.wait_limit > 0 ? a.wait_limit : tc::kWaitPolls;
    init_bars<GROUPS>(bars_of[0]);
  }
  pdl_wait();
  if (warp == 0) tc::tmem_alloc(&s_tmem, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  // no pdl_trigger: what follows, often the pooling pass of the next layer, would take the SMs that this kernel's CTAs leave first and run unevenly
  const uint32_t tmem = s_tmem;
  // One round over the CTA's tiles, and another for marked rows.  body(round's barriers, passes, jobs per tile): job j of tile i has the CTA-wide
  // number i * jobs + j, which picks the S buffer and the softmax group (mod 3).  Every role calls this with its own body; the roles meet at
  // the end of a round.
  int marked = 0;                             // epilogue: this thread has left a row to the second round
  auto rounds = [&](auto body) {
    for (int round = 0, n_pass = redo ? 1 : 2;; ++round, n_pass = 2) {
      marked = 0;
      body(bars_of[round], n_pass, n_pass * n_chunks);
      tc::fence_before_sync();
      if (!__syncthreads_or(marked) || abort_flag->abort) break;
      if (tid == 0) init_bars<GROUPS>(bars_of[1]);
      __syncthreads();
      tc::fence_after_sync();
    }
  };
  // keys of chunk c that belong to its list (a multiple of 32)
  auto keys_of = [&](int c) {
    const int left = c < gathered ? a.p1_blocks * kBS - c * kChunk : (int) n_c - (c - gathered) * kChunk;
    return left < kChunk ? left : kChunk;
  };

  // 640 threads launch with 96 registers each; the warps that issue copies and products leave most of theirs to the others
  if (warp >= 8 && warp < 12) tc::regs_set<Split<GROUPS>::kIssue, Split<GROUPS>::kLaunch>();
  if (warp == 8 || warp == 11) {
    rounds([&](LoopBars& bars, int, int jobs) {
      // ---------------------------------------------------------------- TMA producers: warp 8 Q and keys, warp 11 values
      const bool vals = warp == 11;
      const int first_p2 = jobs - n_chunks;
      uint64_t *full = vals ? bars.v_full : bars.k_full, *empty = vals ? bars.v_empty : bars.k_empty;
      const CUtensorMap *mg = vals ? &maps.vg : &maps.kg, *mc = vals ? &maps.vc : &maps.kc;
      bf16* ring = vals ? sV : sK;
      static_assert(kKStages == kVStages, "one loop for both rings");
      int st = 0;
      uint32_t ph = 1;
      bool ok = true;
      for (int i = 0; ok && i < n_my; ++i) {
        const int tile = blockIdx.x + i * gridDim.x, qs = i & 1;
        const int bh = tile / tiles_per_head, row0 = (tile % tiles_per_head) * kRows;
        if (!vals) {
          if (!(ok = tc::warp_wait(&bars.q_empty[qs], ((i >> 1) & 1) ^ 1, abort_flag))) break;
          tma::expect_tx_w(&bars.q_full[qs], kTile * 2);
          tma::load_4d_w(sQ + qs * kTile, &maps.q, &bars.q_full[qs], 0, row0, bh % a.H, bh / a.H);
        }
        int krow = 0;                                           // lane j: first row of gathered block j
        if (gathered) krow = (int) ((int64_t) bh * a.n1 + p1_block(a, bh, row0 / kBS, min(lane, a.p1_blocks - 1)) * kBS);
        int crow = (int) ((int64_t) bh * n_c);                  // next contiguous chunk
        for (int j = vals ? first_p2 : 0; j < jobs; ++j) {
          const int c = j >= n_chunks ? j - n_chunks : j;
          if (!(ok = tc::warp_wait(&empty[st], ph, abort_flag))) break;
          tma::expect_tx_w(&full[st], kTile * 2);
          if (c < gathered) {
#pragma unroll
            for (int b8 = 0; b8 < 8; ++b8) tma::load_2d_w(ring + st * kTile + b8 * kBS * 64, mg, &full[st], 0, __shfl_sync(0xffffffffu, krow, (c * 8 + b8) & 31));
          } else {
            if (c == gathered) crow = (int) ((int64_t) bh * n_c);
            tma::load_2d_w(ring + st * kTile, mc, &full[st], 0, crow);
            crow += kChunk;
          }
          if (++st == kKStages) { st = 0; ph ^= 1; }
        }
      }
    });
  } else if (warp == 9) {
    rounds([&](LoopBars& bars, int, int jobs) {
      // ---------------------------------------------------------------- MMA issuer 1: S of every job
      {
        const uint32_t id_s = tc::instr_desc(kRows, kChunk, 0, 0);
        const uint32_t hi = (uint32_t) (tc::smem_desc(0, 0, 1024) >> 32);
        auto lo = [](const void* p, uint32_t lbo_bytes) { return ((tc::smem_u32(p) >> 4) & 0x3FFFu) | (((lbo_bytes >> 4) & 0x3FFFu) << 16); };
        constexpr uint32_t kStage = (uint32_t) (kTile * 2) >> 4;
        const uint32_t lQ = lo(sQ, 16), lK = lo(sK, 16);
        int n = 0, ks = 0, buf = 0;                   // jobs issued so far; K ring stage and S buffer of the next one
        uint32_t kph = 0, bph = 0;                    // their phase parities
        bool ok = true;
        for (int i = 0; ok && i < n_my; ++i) {
          const int qs = i & 1;
          if (!(ok = tc::warp_wait(&bars.q_full[qs], (i >> 1) & 1, abort_flag))) break;
          const uint32_t q_ = lQ + qs * kStage;
          for (int j = 0; j < jobs; ++j, ++n) {
            // even lanes: the key chunk; odd lanes: the buffer's previous job (three back), whose group has read S and, in pass 2, P.V P
            const bool b = (lane & 1) && n >= kBufs;
            if (!(ok = tc::warp_wait(b ? &bars.buf_free[buf] : &bars.k_full[ks], b ? bph ^ 1 : kph, abort_flag))) break;
            tc::fence_after_sync();
            const uint32_t k_ = lK + ks * kStage, d = tmem + buf * kChunk;
            tc::umma_ss_k64(d, q_, hi, k_, hi, id_s);
            tc::umma_commit_w(&bars.s_ready[buf]);
            tc::umma_commit_w(&bars.k_empty[ks]);
            if (++ks == kKStages) { ks = 0; kph ^= 1; }
            if (++buf == kBufs) { buf = 0; bph ^= 1; }
          }
          if (!ok) break;
          tc::umma_commit_w(&bars.q_empty[qs]);
        }
      }
    });
  } else if (warp == 10) {
    rounds([&](LoopBars& bars, int, int jobs) {
      // ---------------------------------------------------------------- MMA issuer 2: O (+)= P(job, TMEM) . V chunk
      {
        const uint32_t id_o = tc::instr_desc(kRows, 64, 0, 1);
        const int first_p2 = jobs - n_chunks;
        const uint32_t hi = (uint32_t) (tc::smem_desc(0, 0, 1024) >> 32);
        constexpr uint32_t kStage = (uint32_t) (kTile * 2) >> 4;
        const uint32_t lV = ((tc::smem_u32(sV) >> 4) & 0x3FFFu) | ((1024u >> 4) << 16);
        int vs = 0, buf = 0;
        uint32_t vph = 0, bph = 0;
        bool ok = true;
        for (int i = 0; ok && i < n_my; ++i) {
          for (int j = 0; j < jobs; ++j) {
            // even lanes: the group's job; odd lanes of a pass-2 job: the value chunk; lane 3: O of the tile before the last has been read
            const bool pv = j >= first_p2;
            const int c = j - first_p2;
            uint64_t* bar = &bars.wg_done[buf];
            uint32_t par = bph;
            if (pv && lane == 3 && c == 0 && i > 1) { bar = &bars.o_free[i & 1]; par = ((i - 2) >> 1) & 1; }
            else if (pv && (lane & 1)) { bar = &bars.v_full[vs]; par = vph; }
            if (!(ok = tc::warp_wait(bar, par, abort_flag))) break;
            if (pv) {
              tc::fence_after_sync();
              const uint32_t v_ = lV + vs * kStage, p_ = tmem + buf * kChunk, o_ = tmem + kColO + (i & 1) * 64;
              // P: 16 keys = 8 packed columns per k-step; V: 16 key rows = 2048 bytes
              const int ksteps = keys_of(c) / 16;
              const uint32_t acc = c > 0 ? 1u : 0u;
              if (ksteps >= 4) {
                if (ksteps == 8) tc::umma_ts_k128(o_, p_, v_, hi, id_o, acc);
                else tc::umma_ts_k64(o_, p_, v_, hi, id_o, acc);
              }
              if (ksteps & 2) tc::umma_ts_k32(o_, p_ + (ksteps == 6 ? 32 : 0), v_ + (ksteps == 6 ? 512 : 0), hi, id_o, ksteps == 6 ? 1u : acc);
              tc::umma_commit_w(&bars.v_empty[vs]);
              if (++vs == kVStages) { vs = 0; vph ^= 1; }
            }
            tc::umma_commit_w(&bars.buf_free[buf]);
            if (++buf == kBufs) { buf = 0; bph ^= 1; }
          }
          if (!ok) break;
          tc::umma_commit_w(&bars.o_ready[i & 1]);
        }
      }
    });
  } else if (warp < 8 || warp >= 16) {
    tc::regs_set<Split<GROUPS>::kSoftmax, Split<GROUPS>::kLaunch>();
    rounds([&](LoopBars& bars, int n_pass, int jobs) {
      // ---------------------------------------------------------------- softmax, thread = query row
      const int wg = warp < 8 ? warp >> 2 : 2, qd = warp & 3, r = qd * 32 + lane;
      const int first_p2 = jobs - n_chunks;
      const float sl2 = a.scale * kLog2eF;
      const float lw1 = log2f(a.w1), lw2 = log2f(a.w2);
      const uint32_t t_lane = tmem + ((uint32_t) (qd * 32) << 16);
      int buf = wg;                          // S buffer of this group's next job: it takes every GROUPS-th of the CTA (one of three always meets
      uint32_t bph = 0;                      // the same buffer); the phase parity of that buffer's barriers
      int first = wg;                        // its first job of the tile at hand
      float va[32];
      auto lse_of = [&](int i) {             // the fine part's log-sum-exp of this thread's row of tile i
        const int tile = blockIdx.x + i * gridDim.x;
        return a.lse[(int64_t) (tile / tiles_per_head) * a.Nq + (tile % tiles_per_head) * kRows + r];
      };
      float lse_next = n_pass == 1 && n_my > 0 ? lse_of(0) : 0.f;
      bool ok = true;
      for (int i = 0; ok && i < n_my; ++i) {
        // one pass: the fine part's log-sum-exp is the reference of the exponentials
        float mx = n_pass == 1 ? (REM ? ceilf(lse_next * kLog2eF) + kRefShift : lse_next * kLog2eF) : -INFINITY;
        F2 sum[2] = {f2(0.f, 0.f), f2(0.f, 0.f)};      // four running sums: a chain of adds per element is a third of a job
        if (n_pass == 1 && i + 1 < n_my) lse_next = lse_of(i + 1);
        bool exchanged = n_pass == 1;
        // two passes: the groups exchange their row maxima once per tile, before their first pass-2 job (a group may have none); a copy is
        // rewritten two exchanges later, after every group has passed the barrier in between
        auto exchange_max = [&]() -> bool {
          exchanged = true;
          s_max[i & 1][wg][r] = mx;
          __syncwarp();
          if (lane == 0) tma::mbar_arrive(&bars.xchg);
          const bool ok_ = __all_sync(0xffffffffu, tc::bounded_wait(&bars.xchg, (uint32_t) i & 1, abort_flag));
          mx = fmax3(s_max[i & 1][0][r], s_max[i & 1][1][r], s_max[i & 1][GROUPS - 1][r]);
          if (mx == -INFINITY) mx = 0.f;       // no score above -inf (masked keys): their weight is 0 whatever the reference
          return ok_;
        };
        int j = first;
        for (; j < jobs; j += GROUPS) {
          const bool p2 = j >= first_p2;
          const int c = j >= n_chunks ? j - n_chunks : j;
          const float lw = (c < gathered || !a.two_level) ? lw1 : lw2;
          const int nq = keys_of(c) / 32;
          if (p2 && !exchanged && !(ok = exchange_max())) break;
          ok = __all_sync(0xffffffffu, tc::bounded_wait(&bars.s_ready[buf], bph, abort_flag));
          tc::fence_after_sync();
          if (!ok) break;
          const uint32_t t_s = t_lane + buf * kChunk;
          if (!p2) {
            float m = -INFINITY;
            for (int q4 = 0; q4 < nq; ++q4) {
              tc::tmem_ld32_async(t_s + 32 * q4, va);
              tc::tmem_ld_wait(va);
#pragma unroll
              for (int e = 0; e < 32; e += 2) m = fmax3(m, va[e], va[e + 1]);
            }
            mx = fmaxf(mx, fmaf(m, sl2, lw));
          } else {
            const F2 sl22 = f2(sl2, sl2), off2 = f2(lw - mx, lw - mx);
#pragma unroll 1          // unrolled, the four quarters' registers overlap and spill (to L2: L1 is 28 KB here)
            for (int q4 = 0; q4 < nq; ++q4) {
              tc::tmem_ld32_async(t_s + 32 * q4, va);
              tc::tmem_ld_wait(va);
              uint32_t pk[16];
#pragma unroll
              for (int e = 0; e < 16; ++e) {
                float x0, x1;
                f2_get(f2_fma(f2(va[2 * e], va[2 * e + 1]), sl22, off2), x0, x1);
                x0 = fast_exp2(x0);
                x1 = fast_exp2(x1);
                sum[e & 1] = f2_add(sum[e & 1], f2(x0, x1));
                pk[e] = pack_bf16(x0, x1);
              }
              tc::tmem_st16(t_s + 16 * q4, pk);          // P columns [16 q4, 16 q4 + 16): scores read before
            }
            tc::tmem_st_wait();
          }
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) tma::mbar_arrive(&bars.wg_done[buf]);
          if (GROUPS == kBufs) {
            bph ^= 1;
          } else {
            buf += GROUPS;
            if (buf >= kBufs) { buf -= kBufs; bph ^= 1; }
          }
        }
        first = j - jobs;
        if (ok && !exchanged) ok = exchange_max();
        // the sums of the tile before the last have been read
        if (ok && i > 1) ok = __all_sync(0xffffffffu, tc::bounded_wait(&bars.o_free[i & 1], ((uint32_t) (i - 2) >> 1) & 1, abort_flag));
        if (!ok) break;
        float l0, l1;
        f2_get(f2_add(sum[0], sum[1]), l0, l1);
        s_sum[i & 1][wg][r] = l0 + l1;
        if (wg == 0) s_ref[i & 1][r] = mx;
        __syncwarp();
        if (lane == 0) tma::mbar_arrive(&bars.sum_ready[i & 1]);
      }
    });
  } else {
    tc::regs_set<Split<GROUPS>::kEpilogue, Split<GROUPS>::kLaunch>();
    rounds([&](LoopBars& bars, int n_pass, int jobs) {
      // ---------------------------------------------------------------- epilogue, thread = query row
      const int qd = warp & 3, r = qd * 32 + lane;
      bool ok = true;
      int g0 = 0;                            // the group that takes the tile's first job
      for (int i = 0; i < n_my; ++i) {
        const int tile = blockIdx.x + i * gridDim.x;
        const int bh = tile / tiles_per_head, row = (tile % tiles_per_head) * kRows + r;
        bf16* orow = a.o.row(bh / a.H, bh % a.H, row);
        float* lse_p = a.lse + (int64_t) bh * a.Nq + row;
        // the fine part of this row, and whether the second round owns it: requested before the waits
        uint4 of[8], rest[4];                // rest: half a row of the remainder
        const uint4* rp = REM ? reinterpret_cast<const uint4*>(a.rem + ((int64_t) bh * a.Nq + row) * kD) : nullptr;
#pragma unroll
        for (int q8 = 0; q8 < 8; ++q8) of[q8] = *reinterpret_cast<const uint4*>(orow + 8 * q8);
        if (REM && AHEAD) {
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) rest[q4] = rp[q4];
        }
        const float lse_f = *lse_p;
        bool mine = true;
        if (redo && n_pass == 2) mine = redo[(int64_t) bh * a.Nq + row] != 0;
        ok = ok && __all_sync(0xffffffffu, tc::bounded_wait(&bars.sum_ready[i & 1], (uint32_t) (i >> 1) & 1, abort_flag));
        ok = ok && __all_sync(0xffffffffu, tc::bounded_wait(&bars.o_ready[i & 1], (uint32_t) (i >> 1) & 1, abort_flag));
        tc::fence_after_sync();
        if (!ok) break;
        // Three sums in the order of the tile's jobs, not of the groups: a row's bits do not depend on where in the CTA's list its tile stands
        float lsum = s_sum[i & 1][0][r] + s_sum[i & 1][1][r];
        if constexpr (GROUPS == 3) {
          const int g1 = g0 == 2 ? 0 : g0 + 1, g2 = g1 == 2 ? 0 : g1 + 1;
          lsum = s_sum[i & 1][g0][r] + s_sum[i & 1][g1][r] + s_sum[i & 1][g2][r];
          g0 = (g0 + jobs) % 3;
        }
        const float mx = s_ref[i & 1][r];
        // one pass: the row is this round's unless its sum left the safe range (false for NaN too): the mark hands it to the second
        if (redo && n_pass == 1) {
          mine = lsum < 1e30f;
          redo[(int64_t) bh * a.Nq + row] = mine ? 0 : 1;
          marked |= !mine;
        }
        const float Lf = lse_f * kLog2eF;                        // fine part, log2 domain
        const float Lp = mx + log2f(lsum);
        const float Lm = fmaxf(Lf, Lp);
        const float ef = fast_exp2(Lf - Lm), ep = fast_exp2(Lp - Lm);
        const float inv = 1.f / (ef + ep);
        const float wf = ef * inv, wp = lsum > 0.f ? ep * inv / lsum : 0.f;      // every exponential may have underflowed
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float va[32];
          if (REM && !AHEAD) {
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) rest[q4] = rp[half * 4 + q4];
          }
          tc::tmem_ld32_async(tmem + kColO + (i & 1) * 64 + half * 32 + ((uint32_t) (qd * 32) << 16), va);
          tc::tmem_ld_wait(va);
          if (half == 1) {                                        // O and the sums are in registers
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tma::mbar_arrive(&bars.o_free[i & 1]);
          }
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            const uint4 f = of[half * 4 + q4];
            auto merged = [&](uint32_t fine, uint32_t left, int e) {
              const float x = REM ? bf16_lo(fine) + bf16_lo(left) : bf16_lo(fine), y = REM ? bf16_hi(fine) + bf16_hi(left) : bf16_hi(fine);
              return pack_bf16(x * wf + va[8 * q4 + e] * wp, y * wf + va[8 * q4 + e + 1] * wp);
            };
            const uint4 left = rest[q4];
            if (REM && AHEAD && half == 0) rest[q4] = rp[4 + q4];      // the second half's, a half ahead
            uint4 w;
            w.x = merged(f.x, left.x, 0);
            w.y = merged(f.y, left.y, 2);
            w.z = merged(f.z, left.z, 4);
            w.w = merged(f.w, left.w, 6);
            if (mine) *reinterpret_cast<uint4*>(orow + half * 32 + 8 * q4) = w;
          }
        }
        if (mine) *lse_p = (Lm + log2f(ef + ep)) * 0.6931471805599453f;
      }
    });
  }
  if (abort_flag->abort) {
    tc::abort_drain();
    if (warp >= 12 && warp < 16) poison_lse(a.lse, blockIdx.x, gridDim.x, n_tiles);
  }
  __syncthreads();
  if (threadIdx.x == 0 && abort_flag->abort && a.status) atomicOr(a.status, (int) LLSA_DEV_WAIT_EXPIRED);
  if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

}  // namespace

// Pooled keys per row if the key-loop kernel applies, else 0.  Up to 32 gathered blocks (one per lane of the producer warp); both lists
// end at multiples of 32 keys (an even top-k; N/16 or N/256 a multiple of 32 where that list is attended to).
int pooled_loop_tc_keys(const AttnP<bf16>& a) {
  const int64_t np = (int64_t) (a.p1_blocks + a.p2_blocks) * kBS;
  if (np == 0 || a.Nq % kRows || (a.p1_blocks * kBS) % 32 || (a.p2_blocks * kBS) % 32) return 0;
  if (a.two_level && a.p1_blocks > 32) return 0;
  return (int) np;
}

// Short lists whose fine part crosses with its remainder take two passes whatever the caller offers: the maximum as reference makes the
// weightiest probability exact, which one pass does not, and a second pass over two chunks is cheap (o's error against fp64 / time of the whole forward:
// one level, N = 2560, B=4 H=6, 160 keys 1.714e-3 and 49.3 us, 1.708e-3 and 51.2; two levels, N = 24576, H=6, 224 keys 1.707e-3 and 81.1, 1.696e-3 and 83.8;
// the one-kernel form 1.706e-3, 1.693e-3).  Beyond that it buys less and costs more: N = 40960, top-16, 416 keys 1.701e-3 and 168 us, 1.694e-3 and 184.
bool pooled_loop_one_pass(const AttnP<bf16>& a) {
  return (a.p1_blocks + a.p2_blocks) * kBS > 2 * kChunk || !remainder_wanted(a, false);
}

int launch_attn_fwd_pooled_loop_tc(const LlsaAttnArgs* g, const AttnP<bf16>& a, int64_t BH, cudaStream_t st) {
  LoopMaps maps;
  memset(&maps, 0, sizeof(maps));
  int rc;
  if ((rc = tma::make_map_bhnd(&maps.q, g->q, kRows))) return rc;
  // chunks of the gathered list (two levels), then of the list every row attends to
  const int64_t n_c = a.two_level ? (int64_t) a.p2_blocks * kBS : a.n1;
  const int gathered = a.two_level ? (a.p1_blocks + 7) / 8 : 0, n_chunks = gathered + (int) ((n_c + kChunk - 1) / kChunk);
  if (gathered) {
    if ((rc = tma::make_map_rows(&maps.kg, a.pk, (uint64_t) BH * a.n1, kBS))) return rc;
    if ((rc = tma::make_map_rows(&maps.vg, a.pv, (uint64_t) BH * a.n1, kBS))) return rc;
  }
  if (n_c) {
    if ((rc = tma::make_map_rows(&maps.kc, a.two_level ? a.pk2 : a.pk, (uint64_t) BH * n_c, kChunk))) return rc;
    if ((rc = tma::make_map_rows(&maps.vc, a.two_level ? a.pv2 : a.pv, (uint64_t) BH * n_c, kChunk))) return rc;
  }
  const int tiles_per_head = (int) (a.Nq / kRows), n_tiles = (int) (BH * tiles_per_head);
  int dev = 0, sms = 148;
  LLSA_CUDA_OK(cudaGetDevice(&dev));
  LLSA_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int grid = n_tiles < sms ? n_tiles : sms;
  const size_t smem = 1024 + (size_t) (2 + kKStages + kVStages) * kTile * sizeof(bf16);
  // AHEAD, for lists with a remainder in one pass on two groups: the epilogue is the pace there, and the remainder's first half row requested with the
  // fine part, ahead of the waits, takes one memory latency out of every tile.  Whole forward in us, without / with: two levels, B=2 H=6 N=49152 288 /
  // 277 (284 before there was a third group), N=40960, 288 keys, 274 / 265, 416 keys, H=5, 167.9 / 168.4.  In two passes it costs: H=5 N=40960, 224 and
  // 256 keys, 126 / 128 and 128 / 131.
  const bool three = (a.p1_blocks + a.p2_blocks) * kBS >= (a.rem ? kThreeGroupKeysRem : kThreeGroupKeys);
  unsigned char* redo = g->fwd_redo && pooled_loop_one_pass(a) ? reinterpret_cast<unsigned char*>(g->fwd_redo->ptr) : nullptr;
  auto kernel = three ? (a.rem ? attn_fwd_pooled_loop_tc_kernel<true, 3> : attn_fwd_pooled_loop_tc_kernel<false, 3>)
                : !a.rem ? attn_fwd_pooled_loop_tc_kernel<false, 2>
                : redo ? attn_fwd_pooled_loop_tc_kernel<true, 2, true> : attn_fwd_pooled_loop_tc_kernel<true, 2>;
  const int threads = three ? Split<3>::kThreads : Split<2>::kThreads;
  LLSA_SMEM_LIMIT_REGS(kernel, smem, three ? Split<3>::kLaunch : 0);
  launch_pdl(kernel, grid, threads, smem, st, a, maps, n_chunks, gathered, n_c, n_tiles, tiles_per_head, redo);
  LLSA_LAUNCH_OK("attn_fwd_pooled_loop_tc_kernel");
  return LLSA_OK;
}

}  // namespace llsa
