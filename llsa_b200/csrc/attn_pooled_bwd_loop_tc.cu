// Pooled part of dQ on tcgen05 for LONG pooled key lists (llsa_l1 at any N; llsa_l2 with more than 64 level-2
// keys): the query-major half of _attn_bwd_res_dqkv (sparse_attention_res_1.py:225-281,
// sparse_attention_res_2.py:287-415) restricted to the pooled keys, with a key loop over 64-key chunks.
//
// Per tile of 128 query rows and per chunk c of its pooled keys:
//     S  = Q  . K_c^T   [128 x 64]  (K = 64 channels)        shared-memory operands
//     dP = dO . V_c^T   [128 x 64]
//     dS = exp2(S*scale*log2e + log2 w - lse) * (dP - delta)              softmax warps, thread = query row; the scale (a power of two)
//                                                                         is applied to dQ
//     dQ += dS . K_c    [128 x 64]  (K = 64 keys)             dS read from TENSOR MEMORY (packed bf16 over S), K_c MN-major
// Two levels: first the gathered level-1 blocks (four to a chunk), then the level-2 keys.  Either list may end inside a chunk (at 32 keys):
// what is loaded behind its end (a repeated block, or another head's rows, infinities and NaN included) goes through the softmax with the rest
// of the row, and the dQ products stop in front of it.
// The final log-sum-exp is known in the backward, so one pass over the chunks suffices.  dQ accumulates in TMEM over
// all chunks of the tile and is then added to the fine part already in dq.
// TMEM columns, chunk number n of the CTA (counted over all its tiles): S, and dS over it, at 64 (n mod 4); dP at [256 + 64 (n mod 2), + 64); dQ of
// tile i at [384 + 64 (i mod 2), + 64).
// Roles (one persistent CTA per SM, 16 warps; warps 8 to 11 run in step, tc05.cuh: umma_ss_k64): warps 8 and 11 = TMA producers (Q, dO per
// tile, 2 stages, and K chunks; V chunks; one ring of 8 pairs, 7 with a remainder), warp 9 issues S and dP, warp 10 dQ, warps 0-3 / 4-7 = two softmax
// warpgroups on alternating chunks, warps 12-15 = epilogue, thread = row: adds dQ to the row.  A softmax thread takes its whole row of S and
// dP into registers at once (which is what the register split is for) and hands the dP buffer back before it begins, so that two dP buffers
// do and S gets four.  The two issuing warps run independently (S / dP of the next tile start while dQ of this one is still being issued); an
// S buffer goes back to the S / dP warp through buf_free, committed behind the dQ instructions that read its dS.
// What bounds it: the loop S, dP -> dS -> dQ, 850 cycles a chunk; the tensor pipe takes 576, copies, products and hand-overs without the softmax
// 745, with its exponentials alone left out 810.  Two levels, B=1 H=6 N=262144: 757 us with three buffers for S and dP together and 32 columns loaded at a time, 680 now; l1, B=2 H=4
// N=16384: 64.5 -> 58.5.  On the old form nothing came of three softmax groups (751), of eight warps a chunk (787), of dP handed over apart
// from S (814); four S buffers and two of dP without the early hand-back made it 825.
// The form with one producer lane, the epilogue in the softmax groups and one dQ accumulator (1,050 us) needed 1,130 cycles a chunk for the
// producer's two waits and two copies and left the tensor pipe idle at every tile boundary.
// Every mbarrier wait is bounded (abort flag; the kernel then ends early and frees its TMEM; dq is left partial).
#include <string.h>

#include <type_traits>

#include "attn.cuh"
#include "mma_frag.cuh"
#include "tc05.cuh"
#include "tma.cuh"

namespace llsa {

namespace {

constexpr int kRows = 128;
constexpr int kCk = 64;                      // keys per chunk
constexpr int kTile = kRows * 64;            // elements of a [128 x 64] bf16 tile (16 KB)
constexpr int kChunkElems = kCk * 64;        // elements of a key chunk (8 KB)
template <bool REM>
constexpr int kRing = REM ? 7 : 8;            // key and value chunks; the remainder's tile takes the place of one pair
constexpr int kThreads = 512;
constexpr int kLaunchRegs = 128, kIssueRegs = 40, kEpilogueRegs = 88, kSoftmaxRegs = 192;     // a thread's, per role: 40 + 88 + 2 x 192 = 4 x 128
static_assert(kIssueRegs + kEpilogueRegs + 2 * kSoftmaxRegs <= 4 * kLaunchRegs, "the takers would wait for good");
// Nothing spills with 56 / 88 / 184 or 48 / 88 / 184 either.  Forward + backward in a graph, us, as it is / 56 / 48: two levels, B=3 H=5 N=5376 138.2 / 138.9 / 139.6,
// H=5 N=40960 top-16 492.2 / 492.2 / 492.2, H=6 N=65536 588.7 / 590.5 / 590.7; one level, B=2 H=4 N=16384 313.6 / 314.0 / 315.4, B=4 H=6 N=4096 162.2 / 162.4 / 161.6.
constexpr float kLog2eF = 1.4426950408889634f;
constexpr int kBufs = 4;                     // S buffers (dS over them)
constexpr uint32_t kColDP = 256, kColDQ = 384;
struct DqMaps {
  CUtensorMap q, d_o;         // [B,H,Nq,64] 4-D, box 128 rows
  CUtensorMap dq, rem;        // [B,H,Nq,64] 4-D; [BH*Nq, 64]; box 32 rows
  CUtensorMap kg, vg;         // gathered level-1 keys / values (two levels): [BH*n1, 64], box 16 rows
  CUtensorMap kc, vc;         // contiguous pooled keys / values: [BH*n, 64], box 64 rows
};

struct DqBars {
  uint64_t q_full[2], q_empty[2], kv_full[8], kv_empty[8], out_full[4][2], rem_full[4];
  uint64_t sdp_ready[kBufs], ds_ready[kBufs], buf_free[kBufs], dp_free[2], dq_ready[2], dq_free[2];
};

// jobs: 64-key chunks per tile; gathered: number of leading chunks that are gathered level-1 blocks; n_c: rows per head of the
// contiguous pooled tensor.  REM: the fine part of dq is the bf16 value in dq plus its remainder in a.rem.
template <bool REM>
__global__ void __launch_bounds__(kThreads, 1)
attn_dq_pooled_loop_tc_kernel(AttnP<bf16> a, const __grid_constant__ DqMaps maps, int jobs, int gathered, int64_t n_c, int n_tiles,
                              int tiles_per_head) {
  constexpr int kStages = kRing<REM>;
  extern __shared__ unsigned char smem_dyn[];
  __shared__ DqBars bars;
  __shared__ uint32_t s_tmem;
  __shared__ tc::WaitCtl s_ctl;
  bf16* base = reinterpret_cast<bf16*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  bf16* sQ = base;                          // [2][128][64]
  bf16* sDO = sQ + 2 * kTile;               // [2][128][64]
  bf16* sK = sDO + 2 * kTile;               // [kStages][64][64]
  bf16* sV = sK + kStages * kChunkElems;    // [kStages][64][64]
  bf16* sOut = sV + kStages * kChunkElems;  // [2][128][64]: dq
  bf16* sRem = sOut + 2 * kTile;            // REM: [128][64]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile tc::WaitCtl* abort_flag = &s_ctl;

  if (tid == 0) {
    s_ctl.abort = 0;
    s_ctl.limit = a.wait_limit > 0 ? a.wait_limit : tc::kWaitPolls;
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&bars.q_full[i], 1);
      tc::mbar_init(&bars.q_empty[i], 1);
    }
    for (int i = 0; i < kBufs; ++i) {
      tc::mbar_init(&bars.sdp_ready[i], 1);
      tc::mbar_init(&bars.ds_ready[i], 4);        // one arrival per warp of the group
      tc::mbar_init(&bars.buf_free[i], 1);
    }
    for (int i = 0; i < kStages; ++i) {
      tc::mbar_init(&bars.kv_full[i], 2);         // both producers
      tc::mbar_init(&bars.kv_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&bars.dq_ready[i], 1);
      tc::mbar_init(&bars.dq_free[i], 4);
      tc::mbar_init(&bars.dp_free[i], 4);
    }
    for (int i = 0; i < 4; ++i) {
      tc::mbar_init(&bars.out_full[i][0], 1);
      tc::mbar_init(&bars.out_full[i][1], 1);
      tc::mbar_init(&bars.rem_full[i], 1);
    }
    tc::fence_mbar_init();
  }
  pdl_wait();
  if (warp == 0) tc::tmem_alloc(&s_tmem, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  pdl_trigger();
  const uint32_t tmem = s_tmem;
  const int n_my = (n_tiles - (int) blockIdx.x + (int) gridDim.x - 1) / (int) gridDim.x;
  // keys of chunk j that belong to its list (a multiple of 32)
  auto keys_of = [&](int j) {
    const int left = j < gathered ? a.p1_blocks * kBS - j * kCk : (int) n_c - (j - gathered) * kCk;
    return left < kCk ? left : kCk;
  };

  // the warps that issue copies and products leave most of their registers to the others
  if (warp >= 8 && warp < 12) tc::regs_set<kIssueRegs, kLaunchRegs>();
  if (warp == 8 || warp == 11) {
    // ---------------------------------------------------------------- TMA producers: warp 8 Q, dO and keys, warp 11 values
    const bool vals = warp == 11;
    const CUtensorMap *mg = vals ? &maps.vg : &maps.kg, *mc = vals ? &maps.vc : &maps.kc;
    bf16* ring = vals ? sV : sK;
    int st = 0;
    uint32_t ph = 1;
    bool ok = true;
    for (int i = 0; ok && i < n_my; ++i) {
      const int tile = blockIdx.x + i * gridDim.x, qs = i & 1;
      const int bh = tile / tiles_per_head, row0 = (tile % tiles_per_head) * kRows;
      if (!vals) {
        if (!(ok = tc::warp_wait(&bars.q_empty[qs], ((i >> 1) & 1) ^ 1, abort_flag))) break;
        tma::expect_tx_w(&bars.q_full[qs], 2 * kTile * 2);
        tma::load_4d_w(sQ + qs * kTile, &maps.q, &bars.q_full[qs], 0, row0, bh % a.H, bh / a.H);
        tma::load_4d_w(sDO + qs * kTile, &maps.d_o, &bars.q_full[qs], 0, row0, bh % a.H, bh / a.H);
      }
      int krow = 0;                                           // lane j: first row of gathered block j
      if (gathered) krow = (int) ((int64_t) bh * a.n1 + p1_block(a, bh, row0 / kBS, min(lane, a.p1_blocks - 1)) * kBS);
      int crow = (int) ((int64_t) bh * n_c);                  // next contiguous chunk
      for (int j = 0; j < jobs; ++j) {
        if (!(ok = tc::warp_wait(&bars.kv_empty[st], ph, abort_flag))) break;
        tma::expect_tx_w(&bars.kv_full[st], kChunkElems * 2);
        if (j < gathered) {
#pragma unroll
          for (int b4 = 0; b4 < 4; ++b4)
            tma::load_2d_w(ring + st * kChunkElems + b4 * kBS * 64, mg, &bars.kv_full[st], 0, __shfl_sync(0xffffffffu, krow, (j * 4 + b4) & 31));
        } else {
          tma::load_2d_w(ring + st * kChunkElems, mc, &bars.kv_full[st], 0, crow);
          crow += kCk;
        }
        if (++st == kStages) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 9) {
    // ---------------------------------------------------------------- MMA issuer 1: S and dP
    {
      const uint32_t id_s = tc::instr_desc(kRows, kCk, 0, 0);
      const uint32_t hi = (uint32_t) (tc::smem_desc(0, 0, 1024) >> 32);
      auto lo = [](const void* p, uint32_t lbo_bytes) { return ((tc::smem_u32(p) >> 4) & 0x3FFFu) | (((lbo_bytes >> 4) & 0x3FFFu) << 16); };
      constexpr uint32_t kQStage = (uint32_t) (kTile * 2) >> 4, kCStage = (uint32_t) (kChunkElems * 2) >> 4;
      const uint32_t lQ = lo(sQ, 16), lDO = lo(sDO, 16), lK = lo(sK, 16), lV = lo(sV, 16);
      int cj = 0, st = 0, buf = 0;                  // chunks issued so far; ring stage and buffer of the next one
      uint32_t par = 0, bph = 0;                    // phase parities of the ring stage and of the buffer
      bool ok = true;
      for (int i = 0; ok && i < n_my; ++i) {
        const int qs = i & 1;
        if (!(ok = tc::warp_wait(&bars.q_full[qs], (i >> 1) & 1, abort_flag))) break;
        const uint32_t q_ = lQ + qs * kQStage, o_ = lDO + qs * kQStage;
        for (int j = 0; j < jobs; ++j) {
          // even lanes: the chunk; lanes 1, 5, ..: the S buffer's previous chunk (four back), whose dQ instructions have read dS; lanes 3, 7, ..:
          // the dP buffer's (two back), which its group has loaded
          const bool b = (lane & 3) == 1 && cj >= kBufs, p = (lane & 3) == 3 && cj >= 2;
          if (!(ok = tc::warp_wait(b ? &bars.buf_free[buf] : p ? &bars.dp_free[cj & 1] : &bars.kv_full[st],
                                   b ? bph ^ 1 : p ? (uint32_t) ((cj >> 1) - 1) & 1 : par, abort_flag))) break;
          tc::fence_after_sync();
          const uint32_t d = tmem + buf * 64, dp = tmem + kColDP + (cj & 1) * 64;
          const uint32_t k_ = lK + st * kCStage, v_ = lV + st * kCStage;
          tc::umma_ss_k64(d, q_, hi, k_, hi, id_s);
          tc::umma_ss_k64(dp, o_, hi, v_, hi, id_s);
          tc::umma_commit_w(&bars.sdp_ready[buf]);
          ++cj;
          if (++st == kStages) { st = 0; par ^= 1; }
          if (++buf == kBufs) { buf = 0; bph ^= 1; }
        }
        if (!ok) break;
        tc::umma_commit_w(&bars.q_empty[qs]);
      }
    }
  } else if (warp == 10) {
    // ---------------------------------------------------------------- MMA issuer 2: dQ (+)= dS(chunk, TMEM) . K chunk
    {
      const uint32_t id_dq = tc::instr_desc(kRows, 64, 0, 1);
      const uint32_t hi = (uint32_t) (tc::smem_desc(0, 0, 1024) >> 32);
      constexpr uint32_t kCStage = (uint32_t) (kChunkElems * 2) >> 4;
      const uint32_t lKm = ((tc::smem_u32(sK) >> 4) & 0x3FFFu) | ((1024u >> 4) << 16);
      int st = 0, buf = 0;
      uint32_t bph = 0;
      bool ok = true;
      for (int i = 0; ok && i < n_my; ++i) {
        for (int j = 0; j < jobs; ++j) {
          // odd lanes, first chunk of a tile: dQ of the tile before the last has been read
          const bool f = (lane & 1) && j == 0 && i > 1;
          if (!(ok = tc::warp_wait(f ? &bars.dq_free[i & 1] : &bars.ds_ready[buf], f ? ((uint32_t) (i - 2) >> 1) & 1 : bph, abort_flag))) break;
          tc::fence_after_sync();
          const uint32_t k_ = lKm + st * kCStage, d_ = tmem + buf * 64;       // 16 key rows = 2048 bytes per k-step
          if (keys_of(j) == kCk) tc::umma_ts_k64(tmem + kColDQ + (i & 1) * 64, d_, k_, hi, id_dq, j > 0 ? 1u : 0u);
          else tc::umma_ts_k32(tmem + kColDQ + (i & 1) * 64, d_, k_, hi, id_dq, j > 0 ? 1u : 0u);
          tc::umma_commit_w(&bars.kv_empty[st]);
          tc::umma_commit_w(&bars.buf_free[buf]);
          if (++st == kStages) st = 0;
          if (++buf == kBufs) { buf = 0; bph ^= 1; }
        }
        if (!ok) break;
        tc::umma_commit_w(&bars.dq_ready[i & 1]);
      }
    }
  } else if (warp < 8) {
    tc::regs_set<kSoftmaxRegs, kLaunchRegs>();
    // ---------------------------------------------------------------- dS; thread = query row
    const int wg = warp >> 2, qd = warp & 3, r = qd * 32 + lane;
    const float sl2 = a.scale * kLog2eF;
    const float lw1 = log2f(a.w1), lw2 = log2f(a.w2);
    const uint32_t t_lane = tmem + ((uint32_t) (qd * 32) << 16);
    int buf = wg;                          // this group takes every other chunk: buffer and phase parity of its next one
    uint32_t bph = 0;
    float vs[32], vs2[32], vd[32], vd2[32];
    float lse_next = 0.f, delta_next = 0.f;
    auto fetch = [&](int i) {              // this thread's row of tile i
      const int tile = blockIdx.x + i * gridDim.x;
      const int64_t at = (int64_t) (tile / tiles_per_head) * a.Nq + (tile % tiles_per_head) * kRows + r;
      lse_next = a.lse[at];
      delta_next = a.delta[at];
    };
    if (n_my > 0) fetch(0);
    bool ok = true;
    for (int i = 0; ok && i < n_my; ++i) {
      const float L = lse_next * kLog2eF;
      const F2 nd2 = f2(-delta_next, -delta_next), sl22 = f2(sl2, sl2);
      if (i + 1 < n_my) fetch(i + 1);
      for (int j = (int) ((wg - (int64_t) i * jobs) & 1); j < jobs; j += 2) {
        const float off = ((j < gathered || !a.two_level) ? lw1 : lw2) - L;
        const F2 off2 = f2(off, off);
        ok = __all_sync(0xffffffffu, tc::bounded_wait(&bars.sdp_ready[buf], bph, abort_flag));
        tc::fence_after_sync();
        if (!ok) break;
        const uint32_t t_b = t_lane + buf * 64, t_p = t_lane + kColDP + wg * 64;
        tc::tmem_ld32_async(t_p, vd);
        tc::tmem_ld32_async(t_p + 32, vd2);
        tc::tmem_ld32_async(t_b, vs);
        tc::tmem_ld32_async(t_b + 32, vs2);
        tc::tmem_ld_wait(vd);
        tc::tmem_ld_wait(vd2);
        tc::tmem_ld_wait(vs);
        tc::tmem_ld_wait(vs2);
        tc::fence_before_sync();                     // dP is in registers: the next but one chunk's may come
        __syncwarp();
        if (lane == 0) tma::mbar_arrive(&bars.dp_free[wg]);
        auto ds_of = [&](uint32_t at, const float (&s)[32], const float (&d)[32]) {
          uint32_t pk[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            float x0, x1;
            f2_get(f2_fma(f2(s[2 * e], s[2 * e + 1]), sl22, off2), x0, x1);
            f2_get(f2_mul(f2(fast_exp2(x0), fast_exp2(x1)), f2_add(f2(d[2 * e], d[2 * e + 1]), nd2)), x0, x1);
            pk[e] = pack_bf16(x0, x1);
          }
          tc::tmem_st16(at, pk);
        };
        ds_of(t_b, vs, vd);                          // dS over S; where the list ends after 32 keys, the products stop there
        ds_of(t_b + 16, vs2, vd2);
        tc::tmem_st_wait();
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tma::mbar_arrive(&bars.ds_ready[buf]);
        buf += 2;
        if (buf >= kBufs) { buf -= kBufs; bph ^= 1; }
      }
    }
  } else {
    tc::regs_set<kEpilogueRegs, kLaunchRegs>();
    // ---------------------------------------------------------------- dq += dQ; thread = query row
    // A warp's 32 rows of dq (and of the remainder) come by TMA a tile ahead and leave by TMA from the same memory.  As loads and stores of 16 bytes a
    // lane, 128 bytes apart, they took the epilogue longer than a tile of a few chunks lasts: kernel at three chunks with a remainder (two levels, B=3 H=5
    // N=5376) 21.4 us, now 17.5, at seven (H=5 N=40960, top-16) 47.2 / 45.9, at four without (one level, B=4 H=6 N=4096) 22.6 / 21.4; long lists 668 / 666.
    const int w = warp & 3, r = w * 32 + lane;
    const uint32_t out_row = tc::smem_u32(sOut) + (uint32_t) r * 128 + ((r & 7) << 4), rem_row = out_row + 2 * kTile * 2;      // the row's first chunk, swizzled
    auto request = [&](int i) {              // dq of tile i into stage i & 1
      const int tile = blockIdx.x + i * gridDim.x, bh = tile / tiles_per_head;
      tma::expect_tx_w(&bars.out_full[w][i & 1], 32 * 128);
      tma::load_4d_w(sOut + (i & 1) * kTile + w * 32 * 64, &maps.dq, &bars.out_full[w][i & 1], 0, (tile % tiles_per_head) * kRows + w * 32, bh % a.H, bh / a.H);
    };
    auto request_rem = [&](int i) {
      const int tile = blockIdx.x + i * gridDim.x;
      tma::expect_tx_w(&bars.rem_full[w], 32 * 128);
      tma::load_2d_w(sRem + w * 32 * 64, &maps.rem, &bars.rem_full[w], 0, tile * kRows + w * 32);
    };
    if (n_my > 0) {
      request(0);
      if (REM) request_rem(0);
    }
    bool ok = true;
    for (int i = 0; ok && i < n_my; ++i) {
      const int tile = blockIdx.x + i * gridDim.x, bh = tile / tiles_per_head, row0 = (tile % tiles_per_head) * kRows;
      const uint32_t out = out_row + (i & 1) * (kTile * 2), t_q = tmem + kColDQ + (i & 1) * 64 + ((uint32_t) (w * 32) << 16);
      ok = tc::warp_wait(lane & 1 ? &bars.out_full[w][i & 1] : &bars.dq_ready[i & 1], (uint32_t) (i >> 1) & 1, abort_flag);
      ok = ok && (!REM || tc::warp_wait(&bars.rem_full[w], (uint32_t) i & 1, abort_flag));
      tc::fence_after_sync();
      if (!ok) break;
      if (i + 1 < n_my) {
        tma::reduce_wait_read();             // the last tile has left the other stage
        __syncwarp();
        request(i + 1);
      }
      float v[16];
      auto sum = [&](auto tag, int e) {      // chunk C of the row, eight channels: v[e ..]
        constexpr int C = decltype(tag)::value;
        uint32_t f[4], l[4] = {0u, 0u, 0u, 0u};
        lds128<0>(f[0], f[1], f[2], f[3], out ^ (16 * C));
        if (REM) lds128<0>(l[0], l[1], l[2], l[3], rem_row ^ (16 * C));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float x = REM ? bf16_lo(f[k]) + bf16_lo(l[k]) : bf16_lo(f[k]), y = REM ? bf16_hi(f[k]) + bf16_hi(l[k]) : bf16_hi(f[k]);
          f[k] = pack_bf16(fmaf(v[e + 2 * k], a.scale, x), fmaf(v[e + 2 * k + 1], a.scale, y));
        }
        tc::sts128_xor<16 * C>(out, f[0], f[1], f[2], f[3]);
      };
      tc::tmem_ld16(t_q, v);
      sum(std::integral_constant<int, 0>{}, 0); sum(std::integral_constant<int, 1>{}, 8);
      tc::tmem_ld16(t_q + 16, v);
      sum(std::integral_constant<int, 2>{}, 0); sum(std::integral_constant<int, 3>{}, 8);
      tc::tmem_ld16(t_q + 32, v);
      sum(std::integral_constant<int, 4>{}, 0); sum(std::integral_constant<int, 5>{}, 8);
      tc::tmem_ld16(t_q + 48, v);
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tma::mbar_arrive(&bars.dq_free[i & 1]);
      sum(std::integral_constant<int, 6>{}, 0); sum(std::integral_constant<int, 7>{}, 8);
      tc::fence_async_smem();
      __syncwarp();
      tma::store_4d_w(&maps.dq, 0, row0 + w * 32, bh % a.H, bh / a.H, tc::smem_u32(sOut + (i & 1) * kTile + w * 32 * 64));
      tma::reduce_commit_w();
      if (REM && i + 1 < n_my) request_rem(i + 1);
    }
    tma::reduce_wait_all();                  // dq is in memory before the kernel ends
  }
  if (abort_flag->abort) tc::abort_drain();
  tc::fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && abort_flag->abort && a.status) atomicOr(a.status, (int) LLSA_DEV_WAIT_EXPIRED);
  if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

}  // namespace

// Pooled keys per row if the key-loop dQ kernel applies, else 0: the key-loop forward's range.
int pooled_dq_loop_tc_keys(const AttnP<bf16>& a) { return pooled_loop_tc_keys(a); }

int launch_attn_dq_pooled_loop_tc(const LlsaAttnArgs* g, const AttnP<bf16>& a, int64_t BH, cudaStream_t st) {
  DqMaps maps;
  memset(&maps, 0, sizeof(maps));
  int rc;
  if ((rc = tma::make_map_bhnd(&maps.q, g->q, kRows))) return rc;
  if ((rc = tma::make_map_bhnd(&maps.d_o, g->d_o, kRows))) return rc;
  if ((rc = tma::make_map_bhnd(&maps.dq, g->dq, 32))) return rc;
  if (a.rem && (rc = tma::make_map_rows(&maps.rem, a.rem, (uint64_t) BH * a.Nq, 32))) return rc;
  const int64_t n_c = a.two_level ? (int64_t) a.p2_blocks * kBS : a.n1;
  const int gathered = a.two_level ? (a.p1_blocks + 3) / 4 : 0, jobs = gathered + (int) ((n_c + kCk - 1) / kCk);
  if (gathered) {
    if ((rc = tma::make_map_rows(&maps.kg, a.pk, (uint64_t) BH * a.n1, kBS))) return rc;
    if ((rc = tma::make_map_rows(&maps.vg, a.pv, (uint64_t) BH * a.n1, kBS))) return rc;
  }
  if (n_c) {
    if ((rc = tma::make_map_rows(&maps.kc, a.two_level ? a.pk2 : a.pk, (uint64_t) BH * n_c, kCk))) return rc;
    if ((rc = tma::make_map_rows(&maps.vc, a.two_level ? a.pv2 : a.pv, (uint64_t) BH * n_c, kCk))) return rc;
  }
  const int tiles_per_head = (int) (a.Nq / kRows), n_tiles = (int) (BH * tiles_per_head);
  int dev = 0, sms = 148;
  LLSA_CUDA_OK(cudaGetDevice(&dev));
  LLSA_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int grid = n_tiles < sms ? n_tiles : sms;
  const size_t smem = 1024 + (size_t) (6 * kTile + 2 * (a.rem ? kRing<true> : kRing<false>) * kChunkElems + (a.rem ? kTile : 0)) * sizeof(bf16);
  auto kernel = a.rem ? attn_dq_pooled_loop_tc_kernel<true> : attn_dq_pooled_loop_tc_kernel<false>;
  LLSA_SMEM_LIMIT_REGS(kernel, smem, kLaunchRegs);
  launch_pdl(kernel, grid, kThreads, smem, st, a, maps, jobs, gathered, n_c, n_tiles, tiles_per_head);
  LLSA_LAUNCH_OK("attn_dq_pooled_loop_tc_kernel");
  return LLSA_OK;
}

}  // namespace llsa
