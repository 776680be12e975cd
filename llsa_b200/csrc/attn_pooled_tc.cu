// Pooled stages of the LLSA forward on the 5th-generation tensor cores: TMA loads,
// tcgen05.mma with accumulators in tensor memory (TMEM), warp-specialised and persistent.
//
// Every query row of a parent block attends to the SAME pooled keys: the children of the
// level-2 blocks its parent selected plus all level-2 keys (two levels), or all level-1
// keys (one level) -- sparse_attention_res_2.py:94-149, sparse_attention_res_1.py:85-106.
// That part of the attention is a dense [128 query rows] x [NP pooled keys] problem per
// tile, the shape tcgen05.mma is made for; the private 16-row fine blocks stay on
// mma.sync (attn_fwd_mma.cu: attn_fwd_fine_kernel) and the two parts are merged here
// through their log-sum-exp.
//
// attn_fwd_pooled_tc_kernel: one persistent CTA per SM walks tiles of 128 query rows.  16 warps; 8 to 11 run in step (tc05.cuh: umma_ss_k64):
//   warps 8, 11     : TMA producers.  Per tile Q [128x64] and pooled K [NPx64]; pooled V [NPx64]: 128-byte swizzled tiles in rings of three and two stages.
//   warp 9          : S = Q.PK^T (M=128, N=NP, K=64, both operands from shared memory) into TMEM buffer (tile & 1)
//   warp 10         : O_p = P.PV (M=128, N=64, K=NP) with P read from TENSOR MEMORY (it overwrites the first NP/2 columns of S as packed bf16
//                     pairs) and PV from shared memory, in two parts: all but the last 64 keys as soon as their P is written
//   warps 0-3, 4-7  : two softmax warpgroups on alternate tiles.  Thread r of a group owns query row r = TMEM lane r: reads its NP scores
//                     (tcgen05.ld), softmax in the exp2 domain with +log2(weight) per key class, writes P back (tcgen05.st), leaves the row's
//                     maximum and sum in shared memory and goes on to its next tile
//   warps 12-15     : epilogue, thread = row: merges O_p with the fine part (o, lse written by the fine kernel, requested ahead of the waits) and
//                     stores the final o and lse.  A warp's 32 rows of o come by TMA a tile ahead and leave by TMA from the same memory.
// What bounds it: row maxima, exponentials and hand-overs of the two groups, 3,300 cycles a tile of 192 keys where the special-function units need 1,540, the tensor pipe
// 960 and 48 KB from and to HBM some 2,100.  With producers and issuers that are one lane each, the merge in the softmax groups and o read and written 16
// bytes a lane: two levels, B=8 H=6 N=16384 100.8 us, now 82.4, B=4 62 / 48, B=1 25.3 / 20.4, B=3 H=5 N=5376 (128 keys) 20.4 / 16.5; with the roles as
// here and o still read and written by the epilogue's lanes 92.7 and 22.8.
// All mbarrier waits are bounded; a wait that expires raises a CTA-wide abort flag, every
// role leaves its loop, lse of every row of the CTA becomes NaN (poison_lse) and TMEM is freed.
#include <string.h>

#include <type_traits>

#include "attn.cuh"
#include "mma_frag.cuh"
#include "tc05.cuh"
#include "tma.cuh"

namespace llsa {

constexpr int kTcRows = 128;
constexpr int kKeyStages = 3, kValueStages = 2, kOutStages = 3;      // Q and keys; values; o tiles
constexpr int kTcThreads = 512;

struct TcMaps {
  CUtensorMap q;      // [B,H,N,64] 4-D, box 128 rows
  CUtensorMap o;      // [B,H,N,64] 4-D, box 32 rows
  CUtensorMap pk1, pv1;      // two levels: gathered level-1 keys / values [BH*n1, 64], box 16 rows
  CUtensorMap pkc, pvc;      // the keys / values every row attends to: level 2, or level 1 of one level; box 64 rows
};

struct TcBars {
  // a stage's [Q | pooled keys] part and its [pooled values] part fill and drain separately: Q and the keys are free again as soon
  // as S = Q.PK^T has executed, two tiles before the values (free after O = P.PV), so their refill runs that much further ahead
  uint64_t full_k[kKeyStages], empty_k[kKeyStages], full_v[kValueStages], empty_v[kValueStages], out_full[4][kOutStages], s_ready[2], p_head[2], p_ready[2], buf_free[2], o_ready[2], o_free[2];
};

// np: pooled keys per row; p1_keys: how many of them, the first ones, weigh token_weight; n_gather: blocks of 16 keys gathered per parent (two
// levels), the others are contiguous; n_c: rows per head of the contiguous pooled tensor.
__global__ void __launch_bounds__(kTcThreads, 1)
attn_fwd_pooled_tc_kernel(AttnP<bf16> a, const __grid_constant__ TcMaps maps, int p1_keys, int np, int n_gather, int64_t n_c, int n_tiles,
                          int tiles_per_head) {
  extern __shared__ unsigned char smem_dyn[];
  __shared__ TcBars bars;
  __shared__ uint32_t s_tmem;
  __shared__ tc::WaitCtl s_ctl;
  __shared__ float s_max[2][kTcRows], s_sum[2][kTcRows];      // [TMEM buffer][row]
  bf16* base = reinterpret_cast<bf16*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  const int key_elems = (kTcRows + np) * 64, value_elems = np * 64;      // of a stage: Q and keys; values
  bf16* sV = base + kKeyStages * key_elems;
  bf16* sOut = sV + kValueStages * value_elems;               // [kOutStages][128][64]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile tc::WaitCtl* abort_flag = &s_ctl;

  if (tid == 0) {
    s_ctl.abort = 0;
    s_ctl.limit = a.wait_limit > 0 ? a.wait_limit : tc::kWaitPolls;
    for (int i = 0; i < kKeyStages; ++i) { tc::mbar_init(&bars.full_k[i], 1); tc::mbar_init(&bars.empty_k[i], 1); }
    for (int i = 0; i < kValueStages; ++i) { tc::mbar_init(&bars.full_v[i], 1); tc::mbar_init(&bars.empty_v[i], 1); }
    for (int i = 0; i < 4 * kOutStages; ++i) tc::mbar_init(&bars.out_full[0][0] + i, 1);
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&bars.s_ready[i], 1);
      tc::mbar_init(&bars.buf_free[i], 1);
      tc::mbar_init(&bars.o_ready[i], 1);
      tc::mbar_init(&bars.p_ready[i], 4);       // one arrival per warp of the group
      tc::mbar_init(&bars.p_head[i], 4);        // P of all but the last 64 keys is written (np > 64)
      tc::mbar_init(&bars.o_free[i], 4);
    }
    tc::fence_mbar_init();
  }
  pdl_wait();
  if (warp == 0) tc::tmem_alloc(&s_tmem, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  // no pdl_trigger: what follows, often the pooling pass of the next layer, would take the SMs that this kernel's CTAs leave first and run unevenly
  const uint32_t tmem = s_tmem;
  const int n_my = (n_tiles - (int) blockIdx.x + (int) gridDim.x - 1) / (int) gridDim.x;

  if (warp == 8 || warp == 11) {
    // ---------------------------------------------------------------- TMA producers: warp 8 Q and keys, warp 11 values
    const bool vals = warp == 11;
    const CUtensorMap *mg = vals ? &maps.pv1 : &maps.pk1, *mc = vals ? &maps.pvc : &maps.pkc;
    const uint32_t bytes = (uint32_t) (vals ? np * 64 : kTcRows * 64 + np * 64) * 2;
    const int n_boxes = np / 64 - n_gather / 4, n_stages = vals ? kValueStages : kKeyStages;      // contiguous boxes
    // lane j: first row of gathered block j of tile i, requested a tile ahead
    auto block_row = [&](int i) {
      const int tile = blockIdx.x + i * gridDim.x, bh = tile / tiles_per_head, row0 = (tile % tiles_per_head) * kTcRows;
      return lane < n_gather ? (int) ((int64_t) bh * a.n1 + p1_block(a, bh, row0 / kBS, lane) * kBS) : 0;
    };
    int st = 0, next = n_my > 0 ? block_row(0) : 0;
    uint32_t ph = 1;
    for (int i = 0; i < n_my; ++i) {
      const int tile = blockIdx.x + i * gridDim.x, bh = tile / tiles_per_head, row0 = (tile % tiles_per_head) * kTcRows, krow = next;
      if (i + 1 < n_my) next = block_row(i + 1);
      uint64_t* full = vals ? &bars.full_v[st] : &bars.full_k[st];
      if (!tc::warp_wait(vals ? &bars.empty_v[st] : &bars.empty_k[st], ph, abort_flag)) break;
      tma::expect_tx_w(full, bytes);
      bf16* dst = vals ? sV + st * value_elems : base + st * key_elems + kTcRows * 64;
      if (!vals) tma::load_4d_w(dst - kTcRows * 64, &maps.q, full, 0, row0, bh % a.H, bh / a.H);
      for (int j = 0; j < n_gather; ++j) tma::load_2d_w(dst + j * kBS * 64, mg, full, 0, __shfl_sync(0xffffffffu, krow, j));
      dst += n_gather * kBS * 64;
      for (int j = 0; j < n_boxes; ++j) tma::load_2d_w(dst + j * 64 * 64, mc, full, 0, (int) ((int64_t) bh * n_c) + j * 64);
      if (++st == n_stages) { st = 0; ph ^= 1; }
    }
  } else if (warp == 9) {
    // ---------------------------------------------------------------- S = Q.PK^T
    const uint32_t id_s = tc::instr_desc(kTcRows, np, 0, 0);
    const uint32_t hi = (uint32_t) (tc::smem_desc(0, 0, 1024) >> 32);
    const uint32_t l0 = ((tc::smem_u32(base) >> 4) & 0x3FFFu) | ((16u >> 4) << 16), stage = (uint32_t) (key_elems * 2) >> 4;
    constexpr uint32_t kKeys = (uint32_t) (kTcRows * 64 * 2) >> 4;
    int st = 0;
    uint32_t ph = 0;
    for (int i = 0; i < n_my; ++i) {
      // even lanes: Q and keys; odd lanes: P of the buffer's last tile has been read
      const bool b = (lane & 1) && i >= 2;
      if (!tc::warp_wait(b ? &bars.buf_free[i & 1] : &bars.full_k[st], b ? (uint32_t) ((i >> 1) - 1) & 1 : ph, abort_flag)) break;
      tc::fence_after_sync();
      const uint32_t q_ = l0 + st * stage;
      tc::umma_ss_k64(tmem + (i & 1) * 256, q_, hi, q_ + kKeys, hi, id_s);
      tc::umma_commit_w(&bars.s_ready[i & 1]);
      tc::umma_commit_w(&bars.empty_k[st]);          // Q and the keys of this stage are free once S has executed
      if (++st == kKeyStages) { st = 0; ph ^= 1; }
    }
  } else if (warp == 10) {
    // ---------------------------------------------------------------- O = P.PV
    const uint32_t id_o = tc::instr_desc(kTcRows, 64, 0, 1);
    const uint32_t hi = (uint32_t) (tc::smem_desc(0, 0, 1024) >> 32);
    const uint32_t l0 = ((tc::smem_u32(sV) >> 4) & 0x3FFFu) | ((1024u >> 4) << 16), stage = (uint32_t) (value_elems * 2) >> 4;
    const int head = np - 64;                        // keys of the first part: 0, 64 or 128
    int st = 0;
    uint32_t ph = 0;
    for (int i = 0; i < n_my; ++i) {
      const int b = i & 1;
      const uint32_t par = (uint32_t) (i >> 1) & 1, s_ = tmem + b * 256, o_ = s_ + np, v_ = l0 + st * stage;
      // even lanes: P; lanes 1, 5, ..: the values; lanes 3, 7, ..: the buffer's last O has been read
      const bool v = (lane & 3) == 1, f = (lane & 3) == 3 && i >= 2;
      if (!tc::warp_wait(v ? &bars.full_v[st] : f ? &bars.o_free[b] : head ? &bars.p_head[b] : &bars.p_ready[b], v ? ph : f ? par ^ 1 : par, abort_flag)) break;
      tc::fence_after_sync();
      // P: 16 keys = 8 packed columns per k-step; PV: 16 key rows = 2048 bytes
      if (head == 128) tc::umma_ts_k128(o_, s_, v_, hi, id_o, 0);
      else if (head) tc::umma_ts_k64(o_, s_, v_, hi, id_o, 0);
      if (head) {
        if (!tc::warp_wait(&bars.p_ready[b], par, abort_flag)) break;
        tc::fence_after_sync();
      }
      tc::umma_ts_k64(o_, s_ + head / 2, v_ + head * 8, hi, id_o, head ? 1u : 0u);
      tc::umma_commit_w(&bars.o_ready[b]);
      tc::umma_commit_w(&bars.empty_v[st]);
      tc::umma_commit_w(&bars.buf_free[b]);
      if (++st == kValueStages) { st = 0; ph ^= 1; }
    }
  } else if (warp < 8) {
    // ---------------------------------------------------------------- softmax, thread = query row
    const int wg = warp >> 2, r = (warp & 3) * 32 + lane;
    const float sl2 = a.scale * 1.4426950408889634f;
    const float lw1 = log2f(a.w1), lw2 = log2f(a.w2);
    const uint32_t t_s = tmem + wg * 256 + ((uint32_t) ((warp & 3) * 32) << 16);
    float va[32], vb[32];
    for (int i = wg; i < n_my; i += 2) {
      const uint32_t par = (uint32_t) (i >> 1) & 1;
      // `ok` is warp-uniform: the TMEM accesses below are warp-wide instructions
      bool ok = __all_sync(0xffffffffu, tc::bounded_wait(&bars.s_ready[wg], par, abort_flag));
      tc::fence_after_sync();
      if (!ok) break;
      float m1 = -INFINITY, m2 = -INFINITY;
      auto chunk_max = [&](const float (&v)[32], int c0) {
        float m = fmaxf(v[0], v[1]);
#pragma unroll
        for (int j = 2; j < 32; j += 2) m = fmax3(m, v[j], v[j + 1]);
        if (c0 < p1_keys) m1 = fmaxf(m1, m); else m2 = fmaxf(m2, m);
      };
      tc::tmem_ld32_async(t_s, va);
      tc::tmem_ld_wait(va);
#pragma unroll 1
      for (int c0 = 0; c0 < np; c0 += 64) {        // chunk c0+32 is in flight while chunk c0 is reduced
        tc::tmem_ld32_async(t_s + c0 + 32, vb);
        chunk_max(va, c0);
        tc::tmem_ld_wait(vb);
        if (c0 + 64 < np) tc::tmem_ld32_async(t_s + c0 + 64, va);
        chunk_max(vb, c0 + 32);
        if (c0 + 64 < np) tc::tmem_ld_wait(va);
      }
      const float mx = fmaxf(fmaf(m1, sl2, lw1), fmaf(m2, sl2, lw2));
      F2 sum[2] = {f2(0.f, 0.f), f2(0.f, 0.f)};
      const F2 sl22 = f2(sl2, sl2);
      auto chunk_exp = [&](const float (&v)[32], int c0) {
        const float off = (c0 < p1_keys ? lw1 : lw2) - mx;
        const F2 off2 = f2(off, off);
        uint32_t pk[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          float e0, e1;
          f2_get(f2_fma(f2(v[2 * j], v[2 * j + 1]), sl22, off2), e0, e1);
          e0 = fast_exp2(e0);
          e1 = fast_exp2(e1);
          sum[j & 1] = f2_add(sum[j & 1], f2(e0, e1));
          pk[j] = pack_bf16(e0, e1);
        }
        tc::tmem_st16(t_s + (c0 >> 1), pk);       // P columns [c0/2, c0/2+16): scores read long before
      };
      tc::tmem_ld32_async(t_s, va);
      tc::tmem_ld_wait(va);
#pragma unroll 1
      for (int c0 = 0; c0 < np; c0 += 64) {
        tc::tmem_ld32_async(t_s + c0 + 32, vb);
        chunk_exp(va, c0);
        tc::tmem_ld_wait(vb);
        if (c0 + 64 < np) tc::tmem_ld32_async(t_s + c0 + 64, va);
        chunk_exp(vb, c0 + 32);
        if (c0 + 64 < np) tc::tmem_ld_wait(va);
        if (c0 + 128 == np) {                     // everything but the last 64 keys: the first part of O = P.PV may start
          tc::tmem_st_wait();
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) tma::mbar_arrive(&bars.p_head[wg]);
        }
      }
      // the buffer's last maxima and sums have been read
      if (i >= 2 && !__all_sync(0xffffffffu, tc::bounded_wait(&bars.o_free[wg], par ^ 1, abort_flag))) break;
      float l0, l1;
      f2_get(f2_add(sum[0], sum[1]), l0, l1);
      s_max[wg][r] = mx;
      s_sum[wg][r] = l0 + l1;
      tc::tmem_st_wait();
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tma::mbar_arrive(&bars.p_ready[wg]);
    }
  } else {
    // ---------------------------------------------------------------- epilogue, thread = query row
    const int w = warp & 3, r = w * 32 + lane;
    const uint32_t out_row = tc::smem_u32(sOut) + (uint32_t) r * 128 + ((r & 7) << 4);      // this row's first chunk in stage 0, swizzled
    const uint32_t out_warp = tc::smem_u32(sOut) + (uint32_t) w * 32 * 128;
    float lse_next = 0.f;
    // the fine part of tile i: this warp's rows of o into stage i mod 3, this row's log-sum-exp
    auto request = [&](int i, int st) {
      const int tile = blockIdx.x + i * gridDim.x, bh = tile / tiles_per_head, row0 = (tile % tiles_per_head) * kTcRows;
      tma::expect_tx_w(&bars.out_full[w][st], 32 * 128);
      tma::load_4d_w(sOut + (st * kTcRows + w * 32) * 64, &maps.o, &bars.out_full[w][st], 0, row0 + w * 32, bh % a.H, bh / a.H);
      lse_next = a.lse[(int64_t) bh * a.Nq + row0 + r];
    };
    if (n_my > 0) request(0, 0);
    int st = 0;
    uint32_t out_ph = 0;
    for (int i = 0; i < n_my; ++i) {
      const int tile = blockIdx.x + i * gridDim.x, bh = tile / tiles_per_head, row0 = (tile % tiles_per_head) * kTcRows, buf = i & 1;
      const uint32_t par = (uint32_t) (i >> 1) & 1, t_o = tmem + buf * 256 + np + ((uint32_t) (w * 32) << 16), out = out_row + st * (kTcRows * 128);
      const float lse_f = lse_next;
      if (i + 1 < n_my) {
        tma::reduce_wait_read<1>();                  // the tile before the last has left the stage
        __syncwarp();
        request(i + 1, st == kOutStages - 1 ? 0 : st + 1);
      }
      bool ok = __all_sync(0xffffffffu, tc::bounded_wait(&bars.out_full[w][st], out_ph, abort_flag));
      ok = ok && __all_sync(0xffffffffu, tc::bounded_wait(&bars.p_ready[buf], par, abort_flag));      // maximum and sum
      ok = ok && __all_sync(0xffffffffu, tc::bounded_wait(&bars.o_ready[buf], par, abort_flag));
      tc::fence_after_sync();
      if (!ok) break;
      const float mx = s_max[buf][r], lsum = s_sum[buf][r];
      float va[32];
      tc::tmem_ld32_async(t_o, va);
      const float Lf = lse_f * 1.4426950408889634f;            // fine part, log2 domain
      const float Lp = mx + log2f(lsum);
      const float Lm = fmaxf(Lf, Lp);
      const float ef = fast_exp2(Lf - Lm), ep = fast_exp2(Lp - Lm);
      const float inv = 1.f / (ef + ep);
      const float wf = ef * inv, wp = ep * inv / lsum;
      tc::tmem_ld_wait(va);
      auto merge = [&](auto tag, const float (&v)[8]) {          // chunk C of the row: eight channels
        constexpr int C = decltype(tag)::value;
        uint32_t x, y, z, u;
        lds128<0>(x, y, z, u, out ^ (16 * C));
        x = pack_bf16(bf16_lo(x) * wf + v[0] * wp, bf16_hi(x) * wf + v[1] * wp);
        y = pack_bf16(bf16_lo(y) * wf + v[2] * wp, bf16_hi(y) * wf + v[3] * wp);
        z = pack_bf16(bf16_lo(z) * wf + v[4] * wp, bf16_hi(z) * wf + v[5] * wp);
        u = pack_bf16(bf16_lo(u) * wf + v[6] * wp, bf16_hi(u) * wf + v[7] * wp);
        tc::sts128_xor<16 * C>(out, x, y, z, u);
      };
      auto quarter = [&](int q) -> const float (&)[8] { return *reinterpret_cast<const float (*)[8]>(&va[8 * q]); };
      merge(std::integral_constant<int, 0>{}, quarter(0));
      merge(std::integral_constant<int, 1>{}, quarter(1));
      merge(std::integral_constant<int, 2>{}, quarter(2));
      merge(std::integral_constant<int, 3>{}, quarter(3));
      tc::tmem_ld32_async(t_o + 32, va);
      tc::tmem_ld_wait(va);
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tma::mbar_arrive(&bars.o_free[buf]);
      merge(std::integral_constant<int, 4>{}, quarter(0));
      merge(std::integral_constant<int, 5>{}, quarter(1));
      merge(std::integral_constant<int, 6>{}, quarter(2));
      merge(std::integral_constant<int, 7>{}, quarter(3));
      tc::fence_async_smem();
      __syncwarp();
      tma::store_4d_w(&maps.o, 0, row0 + w * 32, bh % a.H, bh / a.H, out_warp + st * (kTcRows * 128));
      tma::reduce_commit_w();
      a.lse[(int64_t) bh * a.Nq + row0 + r] = (Lm + log2f(ef + ep)) * 0.6931471805599453f;
      if (++st == kOutStages) { st = 0; out_ph ^= 1; }
    }
    tma::reduce_wait_all();                          // o is in memory before the kernel ends
  }
  if (abort_flag->abort) {
    tc::abort_drain();
    if (warp >= 12) poison_lse(a.lse, blockIdx.x, gridDim.x, n_tiles);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && abort_flag->abort && a.status) atomicOr(a.status, (int) LLSA_DEV_WAIT_EXPIRED);
  if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

// Number of pooled keys per query row if the tcgen05 kernel can take this problem, else 0.
int pooled_tc_keys(const AttnP<bf16>& a) {
  const int p1_keys = a.p1_blocks * kBS, np = (a.p1_blocks + a.p2_blocks) * kBS;
  if (np < 64 || np > 192 || np % 64 || p1_keys % 32 || (np - p1_keys) % 64) return 0;
  if (a.Nq % kTcRows) return 0;
  return np;
}

int launch_attn_fwd_pooled_tc(const LlsaAttnArgs* g, const AttnP<bf16>& a, int64_t BH, cudaStream_t st) {
  const int np = pooled_tc_keys(a), p1_keys = a.p1_blocks * kBS;
  TcMaps maps;
  memset(&maps, 0, sizeof(maps));
  int rc;
  if ((rc = tma::make_map_bhnd(&maps.q, g->q, kTcRows))) return rc;
  if ((rc = tma::make_map_bhnd(&maps.o, g->o, 32))) return rc;
  const int n_gather = a.two_level ? a.p1_blocks : 0;
  const int64_t n_c = a.two_level ? a.n2 : a.n1;
  if (n_gather) {
    if ((rc = tma::make_map_rows(&maps.pk1, a.pk, (uint64_t) BH * a.n1, kBS))) return rc;
    if ((rc = tma::make_map_rows(&maps.pv1, a.pv, (uint64_t) BH * a.n1, kBS))) return rc;
  }
  if (np > n_gather * kBS) {
    if ((rc = tma::make_map_rows(&maps.pkc, a.two_level ? a.pk2 : a.pk, (uint64_t) BH * n_c, 64))) return rc;
    if ((rc = tma::make_map_rows(&maps.pvc, a.two_level ? a.pv2 : a.pv, (uint64_t) BH * n_c, 64))) return rc;
  }
  const int tiles_per_head = (int) (a.Nq / kTcRows), n_tiles = (int) (BH * tiles_per_head);
  int dev = 0, sms = 148;
  LLSA_CUDA_OK(cudaGetDevice(&dev));
  LLSA_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int grid = n_tiles < sms ? n_tiles : sms;
  const size_t smem = 1024 + (size_t) (kKeyStages * (kTcRows + np) + kValueStages * np + kOutStages * kTcRows) * 64 * sizeof(bf16);
  LLSA_SMEM_LIMIT((attn_fwd_pooled_tc_kernel), smem);
  launch_pdl(attn_fwd_pooled_tc_kernel, grid, kTcThreads, smem, st, a, maps, p1_keys, np, n_gather, n_c, n_tiles, tiles_per_head);
  LLSA_LAUNCH_OK("attn_fwd_pooled_tc_kernel");
  return LLSA_OK;
}

}  // namespace llsa
