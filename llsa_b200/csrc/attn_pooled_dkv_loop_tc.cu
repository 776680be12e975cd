// Pooled-key gradients on tcgen05, the key-major half of the pooled backward, with a loop over the queries.  Two forms:
//   dense    the keys that EVERY query attends to: all level-1 pooled keys of the one-level form (sparse_attention_res_1.py:362-400),
//            all level-2 keys of the two-level form (_attn_bwd_res_dpkv2, sparse_attention_res_2.py:418-489);
//   gathered the level-1 keys of the two-level form: the children of the level-2 blocks a parent selected, met by the parent's 256
//            query rows only (_attn_bwd_res_dpkv1_sparse, sparse_attention_res_2.py:491-575).
//
// A work unit is (head, chunk of 128 pooled keys) -- gathered: (parent, eight of its blocks) -- and a range of the query rows that
// meet it, walked 64 at a time (a job):
//     S^T  = K_c . Q_t^T   [128 keys x 64 queries]  (K = 64 channels)   shared-memory operands
//     dP^T = V_c . dO_t^T  [128 x 64]
//     P^T  = exp2(S^T*scale*log2e + log2 w - lse[q]),  dS^T = P^T * (dP^T - delta[q])     thread = key row; the scale
//            (a power of two) is applied to dK;
//            lse and delta of the 64 query columns sit in shared memory next to the Q / dO tile
//     dV_c += P^T  . dO_t  [128 x 64]  (K = 64 queries)   P^T, dS^T read from TENSOR MEMORY (packed bf16, written over S^T),
//     dK_c += dS^T . Q_t                                   dO_t / Q_t as MN-major operands (the same tiles)
// dK_c, dV_c accumulate in TMEM over the unit's query range and are then written to the fp32 pooled-gradient
// accumulators (scaled by kv_weight / token_weight, the reference's weighting of the pooled dK/dV side): plain stores if
// the unit covers all queries of its head, reductions otherwise.  Rows of a chunk behind the end of its list (which may end at any
// multiple of 32 keys) hold a repeated block or the rows that follow in memory; their results stay in their own rows and are dropped.
// Work split: all (head, chunk, job) triples in that order form one flat list that is cut into gridDim.x equal pieces,
// one per CTA; a piece is one to a few units (it changes unit where it crosses a chunk boundary).
// TMEM columns, job number n of the CTA: S^T, and P^T and dS^T over it (queries 0..31 at 0 and 16, 32..63 at 32 and 48), at 64 (n mod 4); dP^T at
// 256 + 64 (n mod 2), handed back as soon as its group has it in registers; one pair of accumulators dV, dK at 384.
// Roles (one persistent CTA per SM, 16 warps; warps 8 to 11 run in step, tc05.cuh: umma_ss_k64): warps 8 and 11 = TMA producers (K_c, V_c
// per unit in two stages, Q_t per job; dO_t, lse, delta per job; a ring of 8, gathered 4), warp 9 issues S^T and dP^T, warp 10 dV and dK,
// warps 0-3 / 4-7 = two softmax warpgroups on alternating jobs, warps 12-15 write a unit's dV and dK, thread = key row.  Every mbarrier
// wait is bounded (abort flag, TMEM freed).
// What bounds them.  Dense, tensor pipe 768 cycles a job: the loop S^T, dP^T -> P^T, dS^T -> dV, dK, 1,170 cycles; copies, products and hand-overs
// without the softmax 915, with its exponentials alone left out 1,090.  Two levels, B=1 H=6 N=262144: 870 us with three buffers for both and 32
// columns loaded at a time, 835 now; l1, B=2 H=4 N=16384: 85 -> 79.  Three softmax groups change nothing (866), eight warps a job spill (1,165).
// Gathered: the fp32 reductions, 100 M at the same size, and a unit's few jobs.  A unit's results go through shared memory and are added by bulk reductions of
// whole lines (blocks of 16 keys lie together in the accumulators): 251 -> 198 us; top-16, H=5 N=40960 65 -> 51.5; as reductions of 16 bytes a lane they were
// the pace.  With one pair of accumulators and the dense form's four buffers instead of two pairs and two buffers 198 -> 182, 51.5 -> 47.6.
#include <string.h>

#include <type_traits>

#include "attn.cuh"
#include "mma_frag.cuh"
#include "tc05.cuh"
#include "tma.cuh"

namespace llsa {

namespace {

constexpr int kKeys = 128;                   // keys per unit (MMA M)
constexpr int kQ = 64;                       // query rows per job (MMA N)
constexpr int kKeyTile = kKeys * 64;         // elements of the K / V chunk (16 KB)
constexpr int kQTile = kQ * 64;              // elements of a Q / dO job tile (8 KB)
template <bool GATHER>
constexpr int kRing = GATHER ? 4 : 8;        // stages of the Q / dO ring
constexpr int kThreads = 512;
constexpr int kBufs = 4;                     // S^T buffers (P^T and dS^T over them)
constexpr uint32_t kColDP = 256, kColAcc = 384;
constexpr int kLaunchRegs = 128, kIssueRegs = 56, kEpilogueRegs = 88, kSoftmaxRegs = 184;     // a thread's, per role: 56 + 88 + 2 x 184 = 4 x 128
static_assert(kIssueRegs + kEpilogueRegs + 2 * kSoftmaxRegs <= 4 * kLaunchRegs, "the takers would wait for good");
constexpr float kLog2eF = 1.4426950408889634f;

struct KvMaps {
  CUtensorMap q, d_o;         // [B,H,Nq,64] 4-D, box 64 rows
  CUtensorMap k, v;           // contiguous pooled keys / values [BH*n, 64], box 128 rows (gathered: 16 rows)
  CUtensorMap dpk, dpv;       // gathered: the fp32 accumulators [BH*n, 64], box 16 rows x 32 columns
};

struct KvBars {
  uint64_t kv_full[2], kv_empty[2], q_full[8], q_empty[8], sdp_ready[4], pds_ready[4], buf_free[4], dp_free[2], acc_ready, acc_free;
};

// A CTA's piece of the flat job list, walked unit by unit.
struct Piece {
  int64_t f, f_end;           // next flat job, end of the piece
  int jobs_all;               // jobs per (head, chunk): query rows / 64
  int unit, job0, n;          // current unit: (head, chunk) number, first job, job count
  __device__ Piece(int64_t total, int jobs_all_) : jobs_all(jobs_all_), unit(0), job0(0), n(0) {
    f = total * blockIdx.x / gridDim.x;
    f_end = total * (blockIdx.x + 1) / gridDim.x;
  }
  __device__ bool next() {
    f += n;
    if (f >= f_end) return false;
    unit = (int) (f / jobs_all);
    job0 = (int) (f - (int64_t) unit * jobs_all);
    const int64_t left = f_end - f;
    n = left < jobs_all - job0 ? (int) left : jobs_all - job0;
    return true;
  }
};

// n_keys: rows per head of the pooled tensor; jobs_all: 64-row query jobs per unit; n_base: units; chunks: chunks per head, gathered: per
// parent.
template <bool GATHER>
__global__ void __launch_bounds__(kThreads, 1)
attn_dkv_pooled_loop_tc_kernel(AttnP<bf16> a, const __grid_constant__ KvMaps maps, float* __restrict__ dpk, float* __restrict__ dpv,
                               int64_t n_keys, int jobs_all, int n_base, int chunks, float lw_log2, float out_mul) {
  constexpr int kStages = kRing<GATHER>;
  extern __shared__ unsigned char smem_dyn[];
  __shared__ KvBars bars;
  __shared__ uint32_t s_tmem;
  __shared__ tc::WaitCtl s_ctl;
  __shared__ __align__(16) float s_lse[kStages][kQ], s_delta[kStages][kQ];
  bf16* base = reinterpret_cast<bf16*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  bf16* sK = base;                           // [2][128][64]
  bf16* sV = sK + 2 * kKeyTile;              // [2][128][64]
  bf16* sQ = sV + 2 * kKeyTile;              // [kStages][64][64]
  bf16* sDO = sQ + kStages * kQTile;         // [kStages][64][64]
  float* sOut = reinterpret_cast<float*>(sDO + kStages * kQTile);      // GATHER: [dV, dK][columns 0..31, 32..63][128 keys][32], swizzled
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile tc::WaitCtl* abort_flag = &s_ctl;

  if (tid == 0) {
    s_ctl.abort = 0;
    s_ctl.limit = a.wait_limit > 0 ? a.wait_limit : tc::kWaitPolls;
    for (int i = 0; i < 2; ++i) { tc::mbar_init(&bars.kv_full[i], 1); tc::mbar_init(&bars.kv_empty[i], 1); }
    for (int i = 0; i < kStages; ++i) { tc::mbar_init(&bars.q_full[i], 2); tc::mbar_init(&bars.q_empty[i], 1); }
    for (int i = 0; i < kBufs; ++i) {
      tc::mbar_init(&bars.sdp_ready[i], 1);
      tc::mbar_init(&bars.pds_ready[i], 4);
      tc::mbar_init(&bars.buf_free[i], 1);
    }
    for (int i = 0; i < 2; ++i) tc::mbar_init(&bars.dp_free[i], 4);
    tc::mbar_init(&bars.acc_ready, 1);
    tc::mbar_init(&bars.acc_free, 4);
    tc::fence_mbar_init();
  }
  pdl_wait();
  if (warp == 0) tc::tmem_alloc(&s_tmem, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  pdl_trigger();
  const uint32_t tmem = s_tmem;
  const int units_per_head = GATHER ? chunks * (int) a.nq2 : chunks;
  Piece pc((int64_t) n_base * jobs_all, jobs_all);

  // the warps that issue copies and products leave most of their registers to the others
  if (warp >= 8 && warp < 12) tc::regs_set<kIssueRegs, kLaunchRegs>();
  if (warp == 8 || warp == 11) {
    // ---------------------------------------------------------------- TMA producers: warp 8 the unit's keys and Q, warp 11 dO, lse, delta
    const bool second = warp == 11;
    int st = 0;
    uint32_t ph = 1;
    bool ok = true;
    for (int i = 0; ok && pc.next(); ++i) {
      const int bh = pc.unit / units_per_head, u = pc.unit - bh * units_per_head, ks = i & 1;
      const int c = GATHER ? u % chunks : u, q0 = GATHER ? u / chunks * (kBS * kBS) : 0;      // chunk; first query row of the parent
      if (!second) {
        int krow = (int) ((int64_t) bh * n_keys + (int64_t) c * kKeys);
        if (GATHER) krow = (int) ((int64_t) bh * n_keys + p1_block(a, bh, q0 / kBS, min(c * 8 + (lane & 7), a.p1_blocks - 1)) * kBS);      // lane j: block j
        if (!(ok = tc::warp_wait(&bars.kv_empty[ks], ((i >> 1) & 1) ^ 1, abort_flag))) break;
        tma::expect_tx_w(&bars.kv_full[ks], 2 * kKeyTile * 2);
        if (!GATHER) {
          tma::load_2d_w(sK + ks * kKeyTile, &maps.k, &bars.kv_full[ks], 0, krow);
          tma::load_2d_w(sV + ks * kKeyTile, &maps.v, &bars.kv_full[ks], 0, krow);
        } else {
#pragma unroll
          for (int b8 = 0; b8 < 8; ++b8) {
            const int row = __shfl_sync(0xffffffffu, krow, b8);
            tma::load_2d_w(sK + ks * kKeyTile + b8 * kBS * 64, &maps.k, &bars.kv_full[ks], 0, row);
            tma::load_2d_w(sV + ks * kKeyTile + b8 * kBS * 64, &maps.v, &bars.kv_full[ks], 0, row);
          }
        }
      }
      const int hd = bh % a.H, bt = bh / a.H;
      int qrow = q0 + pc.job0 * kQ;
      for (int j = 0; j < pc.n; ++j, qrow += kQ) {
        if (!(ok = tc::warp_wait(&bars.q_empty[st], ph, abort_flag))) break;
        if (!second) {
          tma::expect_tx_w(&bars.q_full[st], kQTile * 2);
          tma::load_4d_w(sQ + st * kQTile, &maps.q, &bars.q_full[st], 0, qrow, hd, bt);
        } else {
          tma::expect_tx_w(&bars.q_full[st], kQTile * 2 + 2 * kQ * 4);
          tma::load_4d_w(sDO + st * kQTile, &maps.d_o, &bars.q_full[st], 0, qrow, hd, bt);
          tma::load_bulk_w(s_lse[st], a.lse + (int64_t) bh * a.Nq + qrow, kQ * 4, &bars.q_full[st]);
          tma::load_bulk_w(s_delta[st], a.delta + (int64_t) bh * a.Nq + qrow, kQ * 4, &bars.q_full[st]);
        }
        if (++st == kStages) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 9) {
    // ---------------------------------------------------------------- MMA issuer 1: S^T and dP^T of every job
    {
      const uint32_t id_s = tc::instr_desc(kKeys, kQ, 0, 0);
      const uint32_t hi = (uint32_t) (tc::smem_desc(0, 0, 1024) >> 32);
      auto lo = [](const void* p, uint32_t lbo_bytes) { return ((tc::smem_u32(p) >> 4) & 0x3FFFu) | (((lbo_bytes >> 4) & 0x3FFFu) << 16); };
      constexpr uint32_t kQStage = (uint32_t) (kQTile * 2) >> 4, kKeyStage = (uint32_t) (kKeyTile * 2) >> 4;
      const uint32_t lK = lo(sK, 16), lV = lo(sV, 16), lQ = lo(sQ, 16), lDO = lo(sDO, 16);
      int cj = 0, buf = 0;                          // jobs issued so far by this CTA; buffer of the next one
      uint32_t bph = 0;                             // phase parity of that buffer's barriers
      bool ok = true;
      for (int i = 0; ok && pc.next(); ++i) {
        const int ks = i & 1;
        if (!(ok = tc::warp_wait(&bars.kv_full[ks], (i >> 1) & 1, abort_flag))) break;
        const uint32_t k_ = lK + ks * kKeyStage, v_ = lV + ks * kKeyStage;
        for (int j = 0; j < pc.n; ++j, ++cj) {
          const int st = cj & (kStages - 1);
          // even lanes: the query tile; lanes 1, 5, ..: the S^T buffer's previous job (kBufs back), whose P^T / dS^T have been read; lanes 3,
          // 7, ..: the dP^T buffer's (two back), which its group has loaded
          const bool b = (lane & 3) == 1 && cj >= kBufs, p = (lane & 3) == 3 && cj >= 2;
          if (!(ok = tc::warp_wait(b ? &bars.buf_free[buf] : p ? &bars.dp_free[cj & 1] : &bars.q_full[st],
                                   b ? bph ^ 1 : p ? (uint32_t) ((cj >> 1) - 1) & 1 : (uint32_t) (cj / kStages) & 1, abort_flag))) break;
          tc::fence_after_sync();
          const uint32_t d = tmem + buf * 64, dp = tmem + kColDP + (cj & 1) * 64, q_ = lQ + st * kQStage, o_ = lDO + st * kQStage;
          tc::umma_ss_k64(d, k_, hi, q_, hi, id_s);
          tc::umma_ss_k64(dp, v_, hi, o_, hi, id_s);
          tc::umma_commit_w(&bars.sdp_ready[buf]);
          if (++buf == kBufs) { buf = 0; bph ^= 1; }
        }
        if (!ok) break;
        tc::umma_commit_w(&bars.kv_empty[ks]);         // the key chunk is only read by these products
      }
    }
  } else if (warp == 10) {
    // ---------------------------------------------------------------- MMA issuer 2: dV (+)= P^T . dO_t, dK (+)= dS^T . Q_t
    {
      const uint32_t id_o = tc::instr_desc(kKeys, 64, 0, 1);
      const uint32_t hi = (uint32_t) (tc::smem_desc(0, 0, 1024) >> 32);
      auto lo = [](const void* p, uint32_t lbo_bytes) { return ((tc::smem_u32(p) >> 4) & 0x3FFFu) | (((lbo_bytes >> 4) & 0x3FFFu) << 16); };
      constexpr uint32_t kQStage = (uint32_t) (kQTile * 2) >> 4;
      const uint32_t lQm = lo(sQ, 1024), lDOm = lo(sDO, 1024);
      int cj = 0, buf = 0;
      uint32_t bph = 0;
      bool ok = true;
      for (int i = 0; ok && pc.next(); ++i) {
        for (int j = 0; j < pc.n; ++j, ++cj) {
          const int st = cj & (kStages - 1);
          // odd lanes, first job of a unit: the results this accumulator held last have been read
          const bool f = (lane & 1) && j == 0 && i >= 1;
          if (!(ok = tc::warp_wait(f ? &bars.acc_free : &bars.pds_ready[buf], f ? (uint32_t) (i - 1) & 1 : bph, abort_flag))) break;
          tc::fence_after_sync();
          // 4 k-steps of 16 query rows (2048 bytes of the MN-major dO / Q tile)
          const uint32_t o_ = lDOm + st * kQStage, q_ = lQm + st * kQStage, b = tmem + buf * 64, acc = tmem + kColAcc;
          // the first 32 queries' P^T, dS^T lie in the buffer's columns 0 and 16, the others' in 32 and 48
          tc::umma_ts_k32(acc, b, o_, hi, id_o, j > 0 ? 1u : 0u);
          tc::umma_ts_k32(acc, b + 32, o_ + 256, hi, id_o, 1u);
          tc::umma_ts_k32(acc + 64, b + 16, q_, hi, id_o, j > 0 ? 1u : 0u);
          tc::umma_ts_k32(acc + 64, b + 48, q_ + 256, hi, id_o, 1u);
          tc::umma_commit_w(&bars.q_empty[st]);
          tc::umma_commit_w(&bars.buf_free[buf]);
          if (++buf == kBufs) { buf = 0; bph ^= 1; }
        }
        if (!ok) break;
        tc::umma_commit_w(&bars.acc_ready);
      }
    }
  } else if (warp < 8) {
    tc::regs_set<kSoftmaxRegs, kLaunchRegs>();
    // ---------------------------------------------------------------- P^T / dS^T; thread = key row
    const int wg = warp >> 2, qd = warp & 3;
    const float sl2 = a.scale * kLog2eF;
    const uint32_t t_lane = tmem + ((uint32_t) (qd * 32) << 16);
    const int64_t total = pc.f_end - pc.f;         // jobs of this CTA
    int buf = wg;                                  // buffer of this group's next job and the phase parity of its barriers
    uint32_t bph = 0;
    float vs[32], vd[32];
    const F2 sl22 = f2(sl2, sl2), nlog2e2 = f2(-kLog2eF, -kLog2eF), lw2 = f2(lw_log2, lw_log2), minus1 = f2(-1.f, -1.f);
    for (int64_t jn = wg; jn < total; jn += 2) {
      const int st = (int) jn & (kStages - 1);
      const bool ok = __all_sync(0xffffffffu, tc::bounded_wait(&bars.sdp_ready[buf], bph, abort_flag));
      tc::fence_after_sync();
      if (!ok) break;
      const uint32_t t_b = t_lane + buf * 64, t_p = t_lane + kColDP + wg * 64;
      // P^T and dS^T of 32 query columns
      auto half_of = [&](int half, const float (&s)[32], const float (&d)[32], uint32_t to_p, uint32_t to_ds) {
        uint32_t pp[16], pd[16];
#pragma unroll
        for (int q4 = 0; q4 < 8; ++q4) {             // 4 query columns at a time: their lse / delta are broadcast reads
          const float4 l4 = *reinterpret_cast<const float4*>(&s_lse[st][32 * half + 4 * q4]);
          const float4 d4 = *reinterpret_cast<const float4*>(&s_delta[st][32 * half + 4 * q4]);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const F2 l2 = e ? f2(l4.z, l4.w) : f2(l4.x, l4.y), d2 = e ? f2(d4.z, d4.w) : f2(d4.x, d4.y);
            const int k = 4 * q4 + 2 * e;
            float x0, x1;
            f2_get(f2_fma(f2(s[k], s[k + 1]), sl22, f2_fma(l2, nlog2e2, lw2)), x0, x1);
            x0 = fast_exp2(x0);
            x1 = fast_exp2(x1);
            pp[2 * q4 + e] = pack_bf16(x0, x1);
            f2_get(f2_mul(f2(x0, x1), f2_fma(d2, minus1, f2(d[k], d[k + 1]))), x0, x1);
            pd[2 * q4 + e] = pack_bf16(x0, x1);
          }
        }
        tc::tmem_st16(to_p, pp);                     // over columns read before
        tc::tmem_st16(to_ds, pd);
      };
      float vs2[32], vd2[32];
      tc::tmem_ld32_async(t_p, vd);
      tc::tmem_ld32_async(t_p + 32, vd2);
      tc::tmem_ld32_async(t_b, vs);
      tc::tmem_ld32_async(t_b + 32, vs2);
      tc::tmem_ld_wait(vd);
      tc::tmem_ld_wait(vd2);
      tc::tmem_ld_wait(vs);
      tc::tmem_ld_wait(vs2);
      tc::fence_before_sync();                     // dP^T is in registers: the next but one job's may come
      __syncwarp();
      if (lane == 0) tma::mbar_arrive(&bars.dp_free[wg]);
      half_of(0, vs, vd, t_b, t_b + 16);
      half_of(1, vs2, vd2, t_b + 32, t_b + 48);
      tc::tmem_st_wait();
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tma::mbar_arrive(&bars.pds_ready[buf]);
      buf += 2;
      if (buf >= kBufs) { buf -= kBufs; bph ^= 1; }
    }
  } else {
    tc::regs_set<kEpilogueRegs, kLaunchRegs>();
    // ---------------------------------------------------------------- results of a unit; thread = key row
    const int qd = warp & 3, r = qd * 32 + lane;
    for (int i = 0; pc.next(); ++i) {
      const int bh = pc.unit / units_per_head, u = pc.unit - bh * units_per_head, c = GATHER ? u % chunks : u;
      // gathered: row in the pooled tensor where this thread's block of keys begins, -1: no block; dense: this thread's key
      int key_row = -1;
      const int64_t key = (int64_t) c * kKeys + r;
      if (GATHER) {
        const int blk = c * 8 + (r >> 4);
        if (blk < a.p1_blocks) key_row = (int) ((int64_t) bh * n_keys + p1_block(a, bh, u / chunks * kBS, blk) * kBS);
      }
      const bool live = key < n_keys, whole = pc.n == jobs_all;      // dense; whole: the unit saw every query of its head, nobody else adds to these rows
      const bool ok = __all_sync(0xffffffffu, tc::bounded_wait(&bars.acc_ready, (uint32_t) i & 1, abort_flag));
      tc::fence_after_sync();
      if (!ok) break;
      const uint32_t t_acc = tmem + kColAcc + ((uint32_t) (qd * 32) << 16);
      if constexpr (GATHER) {
        // Through shared memory: a warp's 32 rows are two blocks, whose 16 x 64 sums are contiguous in the accumulators.
        const int rows[2] = {__shfl_sync(0xffffffffu, key_row, 0), __shfl_sync(0xffffffffu, key_row, 16)};      // below 0: no such block
        tma::reduce_wait_read();                     // the last unit's results have been read
        __syncwarp();
#pragma unroll
        for (int part = 0; part < 4; ++part) {       // dV's columns 0..31 and 32..63, dK's
          float v[32];
          tc::tmem_ld32_async(t_acc + part * 32, v);
          tc::tmem_ld_wait(v);
          if (part == 3) {
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tma::mbar_arrive(&bars.acc_free);
          }
          const float mul = part < 2 ? out_mul : out_mul * a.scale;
          const uint32_t at = tc::smem_u32(sOut + part * kKeys * 32 + r * 32) + ((r & 7) << 4);
          auto put = [&](auto tag) {
            constexpr int C = decltype(tag)::value;
            tc::sts128_xor<16 * C>(at, __float_as_uint(v[4 * C] * mul), __float_as_uint(v[4 * C + 1] * mul), __float_as_uint(v[4 * C + 2] * mul),
                                   __float_as_uint(v[4 * C + 3] * mul));
          };
          put(std::integral_constant<int, 0>{}); put(std::integral_constant<int, 1>{}); put(std::integral_constant<int, 2>{});
          put(std::integral_constant<int, 3>{}); put(std::integral_constant<int, 4>{}); put(std::integral_constant<int, 5>{});
          put(std::integral_constant<int, 6>{}); put(std::integral_constant<int, 7>{});
          tc::fence_async_smem();
          __syncwarp();
#pragma unroll
          for (int b = 0; b < 2; ++b)
            if (rows[b] >= 0)
              tma::reduce_add_2d_w(part < 2 ? &maps.dpv : &maps.dpk, (part & 1) * 32, rows[b], tc::smem_u32(sOut + part * kKeys * 32 + (qd * 32 + b * kBS) * 32));
        }
        tma::reduce_commit_w();
      } else {
#pragma unroll
        for (int part = 0; part < 8; ++part) {
          float v[16];
          tc::tmem_ld16(t_acc + part * 16, v);
          if (part == 7) {
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tma::mbar_arrive(&bars.acc_free);
          }
          const float mul = part < 4 ? out_mul : out_mul * a.scale;
          float* dst = (part < 4 ? dpv : dpk) + ((int64_t) bh * n_keys + key) * kD + (part & 3) * 16;
          if (!live) {
          } else if (whole) {
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4)
              *reinterpret_cast<float4*>(dst + 4 * q4) = make_float4(v[4 * q4] * mul, v[4 * q4 + 1] * mul, v[4 * q4 + 2] * mul, v[4 * q4 + 3] * mul);
          } else {
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) red_add_v4(dst + 4 * q4, v[4 * q4] * mul, v[4 * q4 + 1] * mul, v[4 * q4 + 2] * mul, v[4 * q4 + 3] * mul);
          }
        }
      }
    }
    if (GATHER) tma::reduce_wait_all();              // the sums are in memory, and shared memory is no longer read, before the kernel ends
  }
  if (abort_flag->abort) tc::abort_drain();
  tc::fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && abort_flag->abort && a.status) atomicOr(a.status, (int) LLSA_DEV_WAIT_EXPIRED);
  if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

}  // namespace

// Launches the dense form (level 1 of one level, level 2 of two levels) and, with two levels, the gathered form: all pooled dK/dV of a
// problem the key-loop dQ kernel takes.
int launch_attn_dkv_pooled_loop_tc(const LlsaAttnArgs* g, const AttnP<bf16>& a, int64_t BH, cudaStream_t st) {
  KvMaps maps;
  memset(&maps, 0, sizeof(maps));
  int rc;
  if ((rc = tma::make_map_bhnd(&maps.q, g->q, kQ))) return rc;
  if ((rc = tma::make_map_bhnd(&maps.d_o, g->d_o, kQ))) return rc;
  int dev = 0, sms = 148;
  LLSA_CUDA_OK(cudaGetDevice(&dev));
  LLSA_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const size_t smem = 1024 + (size_t) (4 * kKeyTile + 2 * kRing<false> * kQTile) * sizeof(bf16);
  // one CTA per SM, each with an equal piece of the flat (unit, job) list
  auto grid_of = [&](int64_t total) { return total < sms ? (int) total : sms; };
  const int64_t n_dense = a.two_level ? (int64_t) a.p2_blocks * kBS : a.n1;
  if (n_dense) {
    if ((rc = tma::make_map_rows(&maps.k, a.two_level ? a.pk2 : a.pk, (uint64_t) BH * n_dense, kKeys))) return rc;
    if ((rc = tma::make_map_rows(&maps.v, a.two_level ? a.pv2 : a.pv, (uint64_t) BH * n_dense, kKeys))) return rc;
    const int chunks = (int) ((n_dense + kKeys - 1) / kKeys), jobs = (int) (a.Nq / kQ), units = (int) BH * chunks;
    const float w = a.two_level ? a.w2 : a.w1, kvw = a.two_level ? a.kvw2 : a.kvw1;
    LLSA_SMEM_LIMIT_REGS((attn_dkv_pooled_loop_tc_kernel<false>), smem, kLaunchRegs);
    launch_pdl(attn_dkv_pooled_loop_tc_kernel<false>, grid_of((int64_t) units * jobs), kThreads, smem, st, 
        a, maps, a.two_level ? a.dpk2 : a.dpk, a.two_level ? a.dpv2 : a.dpv, n_dense, jobs, units, chunks, log2f(w), kvw / w);
    LLSA_LAUNCH_OK("attn_dkv_pooled_loop_tc_kernel");
  }
  if (a.two_level) {
    if ((rc = tma::make_map_rows(&maps.k, a.pk, (uint64_t) BH * a.n1, kBS))) return rc;
    if ((rc = tma::make_map_rows(&maps.v, a.pv, (uint64_t) BH * a.n1, kBS))) return rc;
    const int chunks = (a.p1_blocks + 7) / 8, jobs = kBS * kBS / kQ, units = (int) (BH * a.nq2) * chunks;
    if ((rc = tma::make_map_acc(&maps.dpk, a.dpk, (uint64_t) BH * a.n1, kBS))) return rc;
    if ((rc = tma::make_map_acc(&maps.dpv, a.dpv, (uint64_t) BH * a.n1, kBS))) return rc;
    const size_t smem_g = 1024 + (size_t) (4 * kKeyTile + 2 * kRing<true> * kQTile) * sizeof(bf16) + (size_t) 4 * kKeys * 32 * sizeof(float);
    LLSA_SMEM_LIMIT_REGS((attn_dkv_pooled_loop_tc_kernel<true>), smem_g, kLaunchRegs);
    launch_pdl(attn_dkv_pooled_loop_tc_kernel<true>, grid_of((int64_t) units * jobs), kThreads, smem_g, st, a, maps, a.dpk, a.dpv, a.n1, jobs, units, chunks,
                                                                                                 log2f(a.w1), a.kvw1 / a.w1);
    LLSA_LAUNCH_OK("attn_dkv_pooled_loop_tc_kernel<gathered>");
  }
  return LLSA_OK;
}

}  // namespace llsa
