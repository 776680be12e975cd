// Block-sparse LLSA backward on the tensor cores (bf16, D = 64, 16-token blocks).
// Reference: sparse_indices_attn_res_scatter_bwd_v2 (sparse_attention_res_1.py:403-471)
// and sparse_indices_attn_res_scatter_2_2_bwd_v2 (sparse_attention_res_2.py:578-681).
//
// Kernels on mma.sync.m16n8k16 with the operand fragments of mma_frag.cuh.  The first two hold fine and pooled keys together; they run where
// the tcgen05 kernels do not take the pooled ones: switched off (no_tcgen05), or a list that wants `remainder` and has none (dQ only).
//   attn_dq_mma_kernel     one warp per query block: delta = rowsum(o*do) (the
//                          reference's separate _attn_bwd_preprocess pass), then
//                          S, dP and dQ over the fine, pooled-1 and pooled-2 keys.
//                          Pooled K/V tiles are shared by the CTA through shared
//                          memory (cp.async), fine blocks stream from global memory.
//   attn_dkv_pooled_kernel one CTA per group of 16 query blocks (= one parent):
//                          the group's 256 rows of Q and dO (+ lse, delta) are
//                          staged once in shared memory; the warps share out the
//                          pooled key tiles the group attends to, run the transposed
//                          products S^T, dP^T, dV += P^T.dO, dK += dS^T.Q over the
//                          16 query blocks and add the 16x64 results into fp32
//                          accumulators (one red.add per element and group).
//   attn_dq_fine_kernel    the same for the fine blocks alone (the pooled keys then run on
//                          tcgen05)
//   attn_dkv_fine_ring_kernel  the CSR of a head is cut into ranges of equal length (32
//                          entries, buckets of up to that many kept whole), or the lists
//                          of all heads into one span per warp, however skewed the fan-in
//                          is; an entry is S^T, dP^T, then
//                          dV += P^T.dO, dK += dS^T.Q; pieces of longer buckets meet in
//                          a global partial tensor (no atomics), and
//   attn_dkv_finish_kernel sums the pieces; every store folds in the pooling
//                          backward (dk += (dpk[j] + dpk2[j/16]/16)/16), one bf16 store.
// The reference multiplies k by scale into new tensors first (res_1.py:420-422);
// here scale rides in the exp2 argument and in the epilogues.
#include <string.h>

#include <algorithm>
#include <type_traits>

#include "attn.cuh"
#include "mma_frag.cuh"
#include "tc05.cuh"
#include "tma.cuh"

namespace llsa {

constexpr float kLog2e = 1.4426950408889634f;
constexpr int kRingTileBytes = kRingTileElems * (int) sizeof(bf16);

__device__ __forceinline__ float rowfrag_dot(const RowFrag& x, const RowFrag& y) {
  float acc = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    acc = fmaf(bf16_lo(x.r[i]), bf16_lo(y.r[i]), acc);
    acc = fmaf(bf16_hi(x.r[i]), bf16_hi(y.r[i]), acc);
  }
  return acc;
}

// One lane requests a row of 64 fp32 values.
__device__ __forceinline__ void load_row_w(uint32_t dst, const float* src, uint64_t* bar) {
  asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
               "@e cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], 256, [%2];\n\t}" ::"r"(dst), "l"(src),
               "r"(tc::smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void cp_async4_sa(uint32_t sa, const void* gsrc) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sa), "l"(gsrc) : "memory");
}
// One lane requests rows [row, row + 16) of two [B,H,N,64] tensors as neighbouring 2 KB tiles, counted by one barrier whose phase expects
// `bytes` in all.
__device__ __forceinline__ void load_tiles_w(uint32_t dst, const CUtensorMap* m0, const CUtensorMap* m1, uint64_t* bar, int bytes, int row, int h, int b) {
  asm volatile(
      "{\n\t.reg .pred e;\n\t.reg .b32 d;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "add.u32 d, %0, 2048;\n\t"
      "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%3], %8;\n\t"
      "@e cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%7, %4, %5, %6}], [%3];\n\t"
      "@e cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [d], [%2, {%7, %4, %5, %6}], [%3];\n\t"
      "}" ::"r"(dst), "l"(m0), "l"(m1), "r"(tc::smem_u32(bar)), "r"(row), "r"(h), "r"(b), "r"(0), "r"(bytes)
      : "memory");
}

struct DqRow {
  float L0, L1, delta0, delta1;   // lse (log2 domain) and delta of rows g and g+8
};

// dS (bf16, as A registers) of one 16-key block from its S and dP accumulators
__device__ __forceinline__ void dq_ds(float (&s0)[4], float (&s1)[4], const float (&p0)[4], const float (&p1)[4], const DqRow& r, float sl2,
                                      float lw, uint32_t (&da)[4]) {
  // ds = w * exp(s*scale - lse) * (dp - delta)
  s0[0] = fast_exp2(fmaf(s0[0], sl2, lw - r.L0)) * (p0[0] - r.delta0);
  s0[1] = fast_exp2(fmaf(s0[1], sl2, lw - r.L0)) * (p0[1] - r.delta0);
  s0[2] = fast_exp2(fmaf(s0[2], sl2, lw - r.L1)) * (p0[2] - r.delta1);
  s0[3] = fast_exp2(fmaf(s0[3], sl2, lw - r.L1)) * (p0[3] - r.delta1);
  s1[0] = fast_exp2(fmaf(s1[0], sl2, lw - r.L0)) * (p1[0] - r.delta0);
  s1[1] = fast_exp2(fmaf(s1[1], sl2, lw - r.L0)) * (p1[1] - r.delta0);
  s1[2] = fast_exp2(fmaf(s1[2], sl2, lw - r.L1)) * (p1[2] - r.delta1);
  s1[3] = fast_exp2(fmaf(s1[3], sl2, lw - r.L1)) * (p1[3] - r.delta1);
  da[0] = pack_bf16(s0[0], s0[1]); da[1] = pack_bf16(s0[2], s0[3]); da[2] = pack_bf16(s1[0], s1[1]); da[3] = pack_bf16(s1[2], s1[3]);
}

struct GlobalKV {
  const bf16* k;
  const bf16* v;
  int64_t ks, vs;
  float lw;
};

__device__ __forceinline__ GlobalKV global_kv(const AttnP<bf16>& a, int64_t b, int64_t h, int64_t bh, int64_t qb, int gi, int my_fine,
                                              int n_smem_tiles, float lw1, float lw2) {
  GlobalKV r;
  if (gi < a.topk) {
    const int64_t j = __shfl_sync(0xffffffffu, my_fine, gi);
    r.k = a.k.row(b, h, j * kBS); r.v = a.v.row(b, h, j * kBS); r.ks = a.k.sn; r.vs = a.v.sn; r.lw = 0.f;
  } else {
    const int ip = n_smem_tiles + gi - a.topk;
    if (ip < a.p1_blocks) {
      const int64_t off = (bh * a.n1 + p1_block(a, bh, qb, ip) * kBS) * kD;
      r.k = a.pk + off; r.v = a.pv + off; r.lw = lw1;
    } else {
      const int64_t off = (bh * a.n2 + (int64_t) (ip - a.p1_blocks) * kBS) * kD;
      r.k = a.pk2 + off; r.v = a.pv2 + off; r.lw = lw2;
    }
    r.ks = r.vs = kD;
  }
  return r;
}

__device__ __forceinline__ void stage_pooled_tiles_bwd(const AttnP<bf16>& a, int64_t bh, int64_t qb0, int n_tiles, bf16* sk, bf16* sv) {
  for (int c = threadIdx.x; c < n_tiles * kBS * 8; c += blockDim.x) {
    const int tile = c >> 7, row = (c >> 3) & 15, ch = (c & 7) * 8;
    const bf16 *gk, *gv;
    if (tile < a.p1_blocks) {
      const int64_t off = (bh * a.n1 + p1_block(a, bh, qb0, tile) * kBS + row) * kD + ch;
      gk = a.pk + off; gv = a.pv + off;
    } else {
      const int64_t off = (bh * a.n2 + (int64_t) (tile - a.p1_blocks) * kBS + row) * kD + ch;
      gk = a.pk2 + off; gv = a.pv2 + off;
    }
    const int so = (tile * kBS + row) * kSmemPitch + ch;
    cp_async16(sk + so, gk);
    cp_async16(sv + so, gv);
  }
  cp_async_commit();
}

template <int NW>
__global__ void __launch_bounds__(NW * 32, 4) attn_dq_mma_kernel(AttnP<bf16> a, int n_smem_tiles) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  bf16* sk = reinterpret_cast<bf16*>(smem_raw);
  bf16* sv = sk + n_smem_tiles * kBS * kSmemPitch;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int64_t qb0 = (int64_t) blockIdx.x * NW, qb = qb0 + warp, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
  stage_pooled_tiles_bwd(a, bh, qb0, n_smem_tiles, sk, sv);

  const int my_fine = lane < a.topk ? (int) fine_block(a, bh, qb, lane) : 0;
  const float lw1 = log2f(a.w1), lw2 = log2f(a.w2);
  const float sl2 = a.scale * kLog2e;

  RowFrag qlo, qhi, dlo, dhi;
  load_rowfrag(qlo, a.q.row(b, h, qb * kBS + g), t);
  load_rowfrag(qhi, a.q.row(b, h, qb * kBS + g + 8), t);
  load_rowfrag(dlo, a.d_o.row(b, h, qb * kBS + g), t);
  load_rowfrag(dhi, a.d_o.row(b, h, qb * kBS + g + 8), t);
  DqRow row;
  {
    RowFrag olo, ohi;
    load_rowfrag(olo, a.o_in.row(b, h, qb * kBS + g), t);
    load_rowfrag(ohi, a.o_in.row(b, h, qb * kBS + g + 8), t);
    row.delta0 = quad_sum(rowfrag_dot(olo, dlo));
    row.delta1 = quad_sum(rowfrag_dot(ohi, dhi));
  }
  const int64_t rbase = bh * a.Nq + qb * kBS;
  if (t == 0) { a.delta[rbase + g] = row.delta0; a.delta[rbase + g + 8] = row.delta1; }
  row.L0 = a.lse[rbase + g] * kLog2e;
  row.L1 = a.lse[rbase + g + 8] * kLog2e;

  float dq[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j) dq[j][0] = dq[j][1] = dq[j][2] = dq[j][3] = 0.f;

  const int n_pooled = a.p1_blocks + a.p2_blocks;
  const int n_glob = a.topk + (n_pooled - n_smem_tiles);
  {
    GlobalKV r = global_kv(a, b, h, bh, qb, 0, my_fine, n_smem_tiles, lw1, lw2);
    RowFrag k0, k1, v0, v1;
    load_rowfrag(k0, r.k + (int64_t) g * r.ks, t);
    load_rowfrag(k1, r.k + (int64_t) (g + 8) * r.ks, t);
    load_rowfrag(v0, r.v + (int64_t) g * r.vs, t);
    load_rowfrag(v1, r.v + (int64_t) (g + 8) * r.vs, t);
    for (int gi = 0; gi < n_glob; ++gi) {
      const float lw = r.lw;
      float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f}, p0[4] = {0.f, 0.f, 0.f, 0.f}, p1[4] = {0.f, 0.f, 0.f, 0.f};
      mma_rows_x_keys(s0, s1, qlo, qhi, k0, k1);
      mma_rows_x_keys(p0, p1, dlo, dhi, v0, v1);
      uint32_t tk0[8], tk1[8];   // K transposed in registers: the B operand of dQ += dS.K, no second load
#pragma unroll
      for (int i = 0; i < 8; ++i) { tk0[i] = movmatrix_trans(k0.r[i]); tk1[i] = movmatrix_trans(k1.r[i]); }
      if (gi + 1 < n_glob) {
        r = global_kv(a, b, h, bh, qb, gi + 1, my_fine, n_smem_tiles, lw1, lw2);
        load_rowfrag(k0, r.k + (int64_t) g * r.ks, t);
        load_rowfrag(k1, r.k + (int64_t) (g + 8) * r.ks, t);
        load_rowfrag(v0, r.v + (int64_t) g * r.vs, t);
        load_rowfrag(v1, r.v + (int64_t) (g + 8) * r.vs, t);
      }
      uint32_t da[4];
      dq_ds(s0, s1, p0, p1, row, sl2, lw, da);
#pragma unroll
      for (int i = 0; i < 8; ++i) mma_bf16_16816(dq[i], da[0], da[1], da[2], da[3], tk0[i], tk1[i]);
    }
  }
  cp_async_wait_all();
  __syncthreads();
  for (int ip = 0; ip < n_smem_tiles; ++ip) {
    const bf16* tk = sk + ip * kBS * kSmemPitch;
    const bf16* tv = sv + ip * kBS * kSmemPitch;
    RowFrag k0, k1, v0, v1;
    load_rowfrag_smem(k0, tk + g * kSmemPitch, t);
    load_rowfrag_smem(k1, tk + (g + 8) * kSmemPitch, t);
    load_rowfrag_smem(v0, tv + g * kSmemPitch, t);
    load_rowfrag_smem(v1, tv + (g + 8) * kSmemPitch, t);
    float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f}, p0[4] = {0.f, 0.f, 0.f, 0.f}, p1[4] = {0.f, 0.f, 0.f, 0.f};
    mma_rows_x_keys(s0, s1, qlo, qhi, k0, k1);
    mma_rows_x_keys(p0, p1, dlo, dhi, v0, v1);
    uint32_t da[4];
    dq_ds(s0, s1, p0, p1, row, sl2, ip < a.p1_blocks ? lw1 : lw2, da);
    mma_x_rowfrag_t(dq, da[0], da[1], da[2], da[3], k0, k1);
  }
  store_acc_row_t<0>(a.dq.row(b, h, qb * kBS + g), dq, t, a.scale);
  store_acc_row_t<1>(a.dq.row(b, h, qb * kBS + g + 8), dq, t, a.scale);
}

// Fine blocks only (the pooled keys are on the tcgen05 kernels): one warp per query block; the selected K / V blocks go through a per-warp
// ring in shared memory, filled by TMA two blocks ahead, and K is read a second time, transposed, by ldmatrix.  Bound by the gather from
// L2: 4 KB per (query block, selected block), 9.6 TB/s at 8 x 6 slices of 16384 tokens (167 us with the lists transposed beside it, 158 without; 205
// with P and dS, 1 KB per pair, written out for the dK/dV stage).
constexpr int kDqStages = 3;
struct KvMaps {
  CUtensorMap k, v;            // [B,H,N,64] 4-D, box 16 rows
};
// REM: what rounding dq to bf16 leaves over goes to a.rem, for the pooled stage to add (remainder_wanted).  zero: clear the pooled-gradient
// accumulators on the way, a few rows a warp.
template <int NW, bool REM>
__global__ void __launch_bounds__(NW * 32, 4) attn_dq_fine_kernel(AttnP<bf16> a, const __grid_constant__ KvMaps maps, bool zero) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t s_full[NW][kDqStages];
  __shared__ tc::WaitCtl s_ctl[NW];             // a warp's own: the warps of a CTA share nothing
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  constexpr int kStageBytes = 2 * kRingTileBytes;
  const uint32_t ring_sa = ((tc::smem_u32(smem_raw) + 1023u) & ~1023u) + warp * kDqStages * kStageBytes;
  volatile tc::WaitCtl* ctl = &s_ctl[warp];
  if (lane < kDqStages) tc::mbar_init(&s_full[warp][lane], 1);
  if (lane == 0) {
    ctl->abort = 0;
    ctl->limit = a.wait_limit > 0 ? a.wait_limit : tc::kWaitPolls;
  }
  tc::fence_mbar_init();
  __syncwarp();
  pdl_trigger();
  pdl_wait();
  const int64_t qb = (int64_t) blockIdx.x * NW + warp, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
  const int my_fine = lane < a.topk ? (int) fine_block(a, bh, qb, lane) : 0;
  const int n_glob = a.topk;
  int rst = 0;
  auto request = [&](int i) {
    load_tiles_w(ring_sa + rst * kStageBytes, &maps.k, &maps.v, &s_full[warp][rst], 2 * kRingTileBytes, __shfl_sync(0xffffffffu, my_fine, i) * kBS, (int) h, (int) b);
    rst = rst == kDqStages - 1 ? 0 : rst + 1;
  };
#pragma unroll
  for (int s = 0; s < kDqStages - 1; ++s)
    if (s < n_glob) request(s);
  if (zero) {      // lanes 0..15 a row of dpk, 16..31 of dpv
    const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int64_t r = qb; r < a.n1; r += a.nq1) reinterpret_cast<float4*>((lane < 16 ? a.dpk : a.dpv) + (bh * a.n1 + r) * kD)[lane & 15] = none;
    if (a.two_level)
      for (int64_t r = qb; r < a.n2; r += a.nq1) reinterpret_cast<float4*>((lane < 16 ? a.dpk2 : a.dpv2) + (bh * a.n2 + r) * kD)[lane & 15] = none;
  }
  // shared addresses of stage 0: chunks 2t, 2t + 1 of row g (sa_f, sa_f ^ 16; row g + 8 is 1024 bytes on), ldmatrix rows of channels 0..15
  // (sa_m; ^ 32 c: channels 16c..)
  const uint32_t sa_f = ring_sa + g * 128 + (((2 * t) ^ g) << 4);
  const uint32_t sa_m = ring_sa + ((lane & 7) + ((lane >> 3) & 1) * 8) * 128 + (((lane >> 4) ^ (lane & 7)) << 4);
  RowFrag qlo, qhi, dlo, dhi;
  load_rowfrag(qlo, a.q.row(b, h, qb * kBS + g), t);
  load_rowfrag(qhi, a.q.row(b, h, qb * kBS + g + 8), t);
  load_rowfrag(dlo, a.d_o.row(b, h, qb * kBS + g), t);
  load_rowfrag(dhi, a.d_o.row(b, h, qb * kBS + g + 8), t);
  const int64_t rbase = bh * a.Nq + qb * kBS;
  F2 nl0, nl1, nd0, nd1;                        // minus lse (log2 domain) and minus delta of rows g and g + 8, twice
  {
    RowFrag olo, ohi;
    load_rowfrag(olo, a.o_in.row(b, h, qb * kBS + g), t);
    load_rowfrag(ohi, a.o_in.row(b, h, qb * kBS + g + 8), t);
    const float l0 = -a.lse[rbase + g] * kLog2e, l1 = -a.lse[rbase + g + 8] * kLog2e;
    const float d0 = quad_sum(rowfrag_dot(olo, dlo)), d1 = quad_sum(rowfrag_dot(ohi, dhi));
    if (t == 0) { a.delta[rbase + g] = d0; a.delta[rbase + g + 8] = d1; }
    nl0 = f2(l0, l0); nl1 = f2(l1, l1); nd0 = f2(-d0, -d0); nd1 = f2(-d1, -d1);
  }
  const float sl2 = a.scale * kLog2e;
  const F2 sl22 = f2(sl2, sl2);
  float dq[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j) dq[j][0] = dq[j][1] = dq[j][2] = dq[j][3] = 0.f;
  int st = 0, ph = 0;
  bool ok = true;
  for (int gi = 0; gi < n_glob; ++gi) {
    if (!(ok = tc::warp_wait(&s_full[warp][st], ph, ctl))) break;
    const uint32_t so = st * kStageBytes, f0 = sa_f + so, f1 = f0 ^ 16, m0 = sa_m + so;
    float s0[4], s1[4], p0[4], p1[4];
    half_rows_x_keys<0, true>(s0, s1, qlo, qhi, f0);
    half_rows_x_keys<kRingTileBytes, true>(p0, p1, dlo, dhi, f0);
    // Into the stage read last time: its operands were consumed by products already issued.  The time a request keeps its warp passes beside the
    // first half of the score products: B=8 H=6 N=16384 171.8 us in front of them, 167.5 here, 187 behind all of them; B=4 H=6 N=4096 24.4 / 23.6 /
    // 25.2; B=1 H=5 N=40960, top-16 90.5 / 88.5 / 87.6.
    if (gi + kDqStages - 1 < n_glob) request(gi + kDqStages - 1);
    half_rows_x_keys<0, false>(s0, s1, qlo, qhi, f1);
    half_rows_x_keys<kRingTileBytes, false>(p0, p1, dlo, dhi, f1);
    // P = exp2(s * scale * log2(e) - lse), dS / scale = P * (dP - delta)
    uint32_t da[4];
    auto half = [&](float x0, float x1, float y0, float y1, F2 nl, F2 nd) {
      f2_get(f2_fma(f2(x0, x1), sl22, nl), x0, x1);
      f2_get(f2_mul(f2(fast_exp2(x0), fast_exp2(x1)), f2_add(f2(y0, y1), nd)), y0, y1);
      return pack_bf16(y0, y1);
    };
    da[0] = half(s0[0], s0[1], p0[0], p0[1], nl0, nd0);
    da[1] = half(s0[2], s0[3], p0[2], p0[3], nl1, nd1);
    da[2] = half(s1[0], s1[1], p1[0], p1[1], nl0, nd0);
    da[3] = half(s1[2], s1[3], p1[2], p1[3], nl1, nd1);
#pragma unroll
    for (int c = 0; c < 4; ++c) {           // dQ += dS.K: K read transposed, 16 channels at a time
      uint32_t bk[4];
      ldsm_x4_trans<0>(bk[0], bk[1], bk[2], bk[3], m0 ^ (c << 5));
      mma_bf16_16816(dq[2 * c], da[0], da[1], da[2], da[3], bk[0], bk[1]);
      mma_bf16_16816(dq[2 * c + 1], da[0], da[1], da[2], da[3], bk[2], bk[3]);
    }
    if (st == kDqStages - 1) { st = 0; ph ^= 1; } else { ++st; }
  }
  if (!ok) {
    tc::abort_drain();
    if (lane == 0 && a.status) atomicOr(a.status, (int) LLSA_DEV_WAIT_EXPIRED);
    return;
  }
  // the tile leaves through the idle ring (stmatrix, then eight lanes write one whole row)
  __syncwarp();
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    float x[2][4];
    uint32_t w[4];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
#pragma unroll
      for (int e = 0; e < 4; ++e) x[u][e] = dq[2 * c + u][e] * a.scale;
      w[2 * u] = pack_bf16(x[u][0], x[u][1]);
      w[2 * u + 1] = pack_bf16(x[u][2], x[u][3]);
    }
    stsm_x4<0>(sa_m ^ (c << 5), w[0], w[1], w[2], w[3]);
    if (REM)
      stsm_x4<kRingTileBytes>(sa_m ^ (c << 5), pack_rest(x[0][0], x[0][1], w[0]), pack_rest(x[0][2], x[0][3], w[1]),
                              pack_rest(x[1][0], x[1][1], w[2]), pack_rest(x[1][2], x[1][3], w[3]));
  }
  __syncwarp();
  const uint32_t sa_cp = ring_sa + (lane >> 3) * 128 + (((lane & 7) ^ (lane >> 3)) << 4);
  bf16* out = a.dq.row(b, h, qb * kBS + (lane >> 3)) + (lane & 7) * 8;
  const int64_t step = 4 * a.dq.sn;
  uint4 x;
  lds128<0>(x.x, x.y, x.z, x.w, sa_cp);         *reinterpret_cast<uint4*>(out) = x;
  lds128<512>(x.x, x.y, x.z, x.w, sa_cp ^ 64);  *reinterpret_cast<uint4*>(out + step) = x;
  lds128<1024>(x.x, x.y, x.z, x.w, sa_cp);      *reinterpret_cast<uint4*>(out + 2 * step) = x;
  lds128<1536>(x.x, x.y, x.z, x.w, sa_cp ^ 64); *reinterpret_cast<uint4*>(out + 3 * step) = x;
  if (REM) {
    constexpr int TB = kRingTileBytes;
    bf16* rp = a.rem + (rbase + (lane >> 3)) * kD + (lane & 7) * 8;
    lds128<TB>(x.x, x.y, x.z, x.w, sa_cp);             *reinterpret_cast<uint4*>(rp) = x;
    lds128<TB + 512>(x.x, x.y, x.z, x.w, sa_cp ^ 64);  *reinterpret_cast<uint4*>(rp + 4 * kD) = x;
    lds128<TB + 1024>(x.x, x.y, x.z, x.w, sa_cp);      *reinterpret_cast<uint4*>(rp + 8 * kD) = x;
    lds128<TB + 1536>(x.x, x.y, x.z, x.w, sa_cp ^ 64); *reinterpret_cast<uint4*>(rp + 12 * kD) = x;
  }
}

// P^T and dS^T (bf16, as A registers) of one (key tile) x (query block) pair from the
// transposed accumulators: rows = keys (g, g+8), columns = query rows (tile 0: 0..7, tile 1: 8..15).
__device__ __forceinline__ void dkv_p_ds(float (&s0)[4], float (&s1)[4], float (&e0)[4], float (&e1)[4], float2 la, float2 lb, float2 da,
                                         float2 db, float sl2, float lw, uint32_t (&pa)[4], uint32_t (&ea)[4]) {
  const float a0 = lw - la.x * kLog2e, a1 = lw - la.y * kLog2e, b0 = lw - lb.x * kLog2e, b1 = lw - lb.y * kLog2e;
  // c0: (key g, row 2t)  c1: (key g, row 2t+1)  c2: (key g+8, row 2t)  c3: (key g+8, row 2t+1)
  s0[0] = fast_exp2(fmaf(s0[0], sl2, a0)); s0[1] = fast_exp2(fmaf(s0[1], sl2, a1));
  s0[2] = fast_exp2(fmaf(s0[2], sl2, a0)); s0[3] = fast_exp2(fmaf(s0[3], sl2, a1));
  s1[0] = fast_exp2(fmaf(s1[0], sl2, b0)); s1[1] = fast_exp2(fmaf(s1[1], sl2, b1));
  s1[2] = fast_exp2(fmaf(s1[2], sl2, b0)); s1[3] = fast_exp2(fmaf(s1[3], sl2, b1));
  e0[0] = s0[0] * (e0[0] - da.x); e0[1] = s0[1] * (e0[1] - da.y); e0[2] = s0[2] * (e0[2] - da.x); e0[3] = s0[3] * (e0[3] - da.y);
  e1[0] = s1[0] * (e1[0] - db.x); e1[1] = s1[1] * (e1[1] - db.y); e1[2] = s1[2] * (e1[2] - db.x); e1[3] = s1[3] * (e1[3] - db.y);
  pa[0] = pack_bf16(s0[0], s0[1]); pa[1] = pack_bf16(s0[2], s0[3]); pa[2] = pack_bf16(s1[0], s1[1]); pa[3] = pack_bf16(s1[2], s1[3]);
  ea[0] = pack_bf16(e0[0], e0[1]); ea[1] = pack_bf16(e0[2], e0[3]); ea[2] = pack_bf16(e1[0], e1[1]); ea[3] = pack_bf16(e1[2], e1[3]);
}

template <int NW>
__global__ void __launch_bounds__(NW * 32, 1) attn_dkv_pooled_kernel(AttnP<bf16> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  bf16* sq = reinterpret_cast<bf16*>(smem_raw);              // [256][kSmemPitch]
  bf16* sd = sq + kBS * kBS * kSmemPitch;                    // [256][kSmemPitch]
  float* sl = reinterpret_cast<float*>(sd + kBS * kBS * kSmemPitch);   // lse [256]
  float* sdel = sl + kBS * kBS;                                        // delta [256]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int64_t grp = blockIdx.x, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
  const float sl2 = a.scale * kLog2e;
  // stage the group's 256 rows of Q and dO
  const int64_t row0 = grp * kBS * kBS;
  for (int c = threadIdx.x; c < kBS * kBS * 8; c += blockDim.x) {
    const int r = c >> 3, ch = (c & 7) * 8;
    cp_async16(sq + r * kSmemPitch + ch, a.q.row(b, h, row0 + r) + ch);
    cp_async16(sd + r * kSmemPitch + ch, a.d_o.row(b, h, row0 + r) + ch);
  }
  cp_async_commit();
  for (int r = threadIdx.x; r < kBS * kBS; r += blockDim.x) {
    sl[r] = a.lse[bh * a.Nq + row0 + r];
    sdel[r] = a.delta[bh * a.Nq + row0 + r];
  }
  cp_async_wait_all();
  __syncthreads();

  const int ntiles = a.p1_blocks + a.p2_blocks;
  for (int i = warp; i < ntiles; i += NW) {
    const bf16 *kp, *vp;
    float *gk, *gv;
    float lw;
    if (i < a.p1_blocks) {
      const int64_t off = (bh * a.n1 + p1_block(a, bh, grp * kBS, i) * kBS) * kD;
      kp = a.pk + off; vp = a.pv + off; gk = a.dpk + off; gv = a.dpv + off; lw = log2f(a.kvw1);
    } else {
      const int64_t off = (bh * a.n2 + (int64_t) (i - a.p1_blocks) * kBS) * kD;
      kp = a.pk2 + off; vp = a.pv2 + off; gk = a.dpk2 + off; gv = a.dpv2 + off; lw = log2f(a.kvw2);
    }
    RowFrag ka, kb, va, vb;
    load_rowfrag(ka, kp + g * kD, t);
    load_rowfrag(kb, kp + (g + 8) * kD, t);
    load_rowfrag(va, vp + g * kD, t);
    load_rowfrag(vb, vp + (g + 8) * kD, t);
    float dk[8][4], dv[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j) dk[j][0] = dk[j][1] = dk[j][2] = dk[j][3] = dv[j][0] = dv[j][1] = dv[j][2] = dv[j][3] = 0.f;
#pragma unroll 1
    for (int qi = 0; qi < kBS; ++qi) {
      const bf16* tq = sq + qi * kBS * kSmemPitch;
      const bf16* td = sd + qi * kBS * kSmemPitch;
      float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f}, e0[4] = {0.f, 0.f, 0.f, 0.f}, e1[4] = {0.f, 0.f, 0.f, 0.f};
      RowFrag q0, q1, d0, d1;
      load_rowfrag_smem(q0, tq + g * kSmemPitch, t);
      load_rowfrag_smem(q1, tq + (g + 8) * kSmemPitch, t);
      mma_rows_x_keys(s0, s1, ka, kb, q0, q1);
      load_rowfrag_smem(d0, td + g * kSmemPitch, t);
      load_rowfrag_smem(d1, td + (g + 8) * kSmemPitch, t);
      mma_rows_x_keys(e0, e1, va, vb, d0, d1);
      const float2 la = *reinterpret_cast<const float2*>(sl + qi * kBS + 2 * t), lb = *reinterpret_cast<const float2*>(sl + qi * kBS + 8 + 2 * t);
      const float2 da = *reinterpret_cast<const float2*>(sdel + qi * kBS + 2 * t), db = *reinterpret_cast<const float2*>(sdel + qi * kBS + 8 + 2 * t);
      uint32_t pa[4], ea[4];
      dkv_p_ds(s0, s1, e0, e1, la, lb, da, db, sl2, lw, pa, ea);
      // the same tiles, transposed in registers, are the B operands of dV and dK
      mma_x_rowfrag_t(dv, pa[0], pa[1], pa[2], pa[3], d0, d1);
      mma_x_rowfrag_t(dk, ea[0], ea[1], ea[2], ea[3], q0, q1);
    }
    // a lane owns channels [16t, 16t+16) of key rows g and g+8: four 128-bit reductions per row
    red_acc_row_t<0>(gk + g * kD, dk, t, a.scale);
    red_acc_row_t<1>(gk + (g + 8) * kD, dk, t, a.scale);
    red_acc_row_t<0>(gv + g * kD, dv, t, 1.f);
    red_acc_row_t<1>(gv + (g + 8) * kD, dv, t, 1.f);
  }
}

// ---- fine dK/dV: ranges of the CSR entry list, whatever the fan-in ------------------------------
// The CSR of a head lists, bucket after bucket (KV block after KV block), the query blocks that selected each KV
// block.  Fan-in is very uneven (0 ... >150 on correlated inputs), so the work is cut by ENTRIES, not by buckets: the
// index transpose cuts the list into ranges of nominally kRangeEntries entries, one per warp, moving a cut that would
// fall inside a bucket of at most kRangeEntries entries to that bucket's start.  Most buckets are therefore finished
// by one warp; longer ones are cut at multiples of kRangeEntries and their pieces meet in the `partial` scratch (summed in window order by the
// finish kernel).  Small problems are cut into equal spans instead.  No atomics: bit-reproducible.
constexpr int kTileFloats = 64 * 32;            // a parked dK + dV tile pair: 64 accumulators x 32 lanes (8 KB)

__device__ __forceinline__ int64_t csr_off(const AttnP<bf16>& a, int64_t bh, int64_t j) {
  const int64_t o = bh * (a.n1 + 1) + j;
  return a.off64 ? reinterpret_cast<const int64_t*>(a.offsets)[o] : (int64_t) reinterpret_cast<const int32_t*>(a.offsets)[o];
}

// A parked dK + dV tile pair is [16 accumulator quads][32 lanes] float4: every access of a warp is one 128-bit
// instruction over 512 contiguous bytes.  (A warp gets about eight loads per memory round trip, however many it has issued:
// the same tile as 64 32-bit loads cost the finish kernel eight round trips per piece in a clock trace.)
__device__ __forceinline__ void tile_to_mem(float* s, const float (&dk)[8][4], const float (&dv)[8][4], int lane) {
  float4* s4 = reinterpret_cast<float4*>(s) + lane;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    s4[u * 32] = make_float4(dk[u][0], dk[u][1], dk[u][2], dk[u][3]);
    s4[(8 + u) * 32] = make_float4(dv[u][0], dv[u][1], dv[u][2], dv[u][3]);
  }
}
__device__ __forceinline__ void tile_zero(float (&dk)[8][4], float (&dv)[8][4]) {
#pragma unroll
  for (int u = 0; u < 8; ++u) dk[u][0] = dk[u][1] = dk[u][2] = dk[u][3] = dv[u][0] = dv[u][1] = dv[u][2] = dv[u][3] = 0.f;
}

// ---- fine dK/dV kernel ------------------------------------------------------------------------------
// dV_j += P^T.dO and dK_j += dS^T.Q over the query blocks that selected KV block j (reference:
// sparse_attention_res_2.py:371-415, the dK/dV half of _attn_bwd_res_dqkv).
//   * S^T = K.Q^T and dP^T = V.dO^T come out with rows = keys, which is the A operand of the two products that follow: nothing is
//     transposed.  K and V of the bucket stay in registers as A operands.
//   * The Q / dO tiles of an entry come through a per-warp ring of kRingFineStages stages, two entries ahead, as two TMA copies issued
//     by one lane (plus one 4-byte copy per lane: lse and delta); K, V and the pooled-gradient rows of the next bucket through a buffer
//     of their own, requested as soon as those of the bucket at hand sit in registers.
//   * One CTA of twelve warps per SM, in two forms.  Windows (ranges of kRangeEntries, i.e. problems of some 4,700 ranges and more): a window is two
//     ranges, a warp draws one range after another from a counter in shared memory, and where a long bucket crosses from the first range of a
//     window into the second one warp takes both.  All SMs work on neighbouring entries at any time, so that the tiles stay in L2.  Spans (smaller
//     problems, whose tensors L2 holds anyway): the entries of all heads, one head behind the other, are cut into equal spans, one per warp, wherever
//     the cut falls: every warp begins once, and all end together.  As CTAs of four warps, each with a range of 16 entries and its own start, two CTAs
//     an SM, these problems took 63 us instead of 48 (45 now; one level, B=4 H=6 N=4096), 55 / 44 (two levels, B=3 H=5 N=5376), 78 / 60 (one level, B=2
//     H=4 N=16384).
//     Pieces of buckets that straddle windows or spans go to the `partial` scratch and attn_dkv_finish_kernel adds them in order.
// What bounds it: latency.  0.46 instructions per scheduler and cycle: 54 % of the issue slots stay empty with three warps on a scheduler, each on
// one serial chain (wait, S and dP, exponentials, the two products: some 290 instructions per entry); then the raggedness of the last ranges.
// 168 registers, nothing spilled.  With P and dS handed over by the dQ stage instead of recomputed this kernel issued half as much,
// but 1 KB per entry went out to HBM and came back: at 8 x 6 slices of 16384 tokens, top 8, dQ stage 205 -> 158 us and this one 192 -> 255
// on random inputs, 207 -> 164 and 284 -> 255 on correlated ones; at 6 of 262144 421 -> 315 and 563 -> 460 (the first figures of the
// correlated pairs with eight warps per SM in groups of four that waited for the longest of their ranges: 322 and 645 on random inputs).
// Accumulator layout (ldmatrix): tile u holds channels 8u + 2t, 8u + 2t + 1 of keys g (c0, c1) and g + 8 (c2, c3).
constexpr int kRingWarps = 12;                  // warps per CTA, one CTA per SM
constexpr int kRingFineStages = 3;
constexpr int kRingFineStageBytes = 2 * kRingTileBytes;                                // Q tile, dO tile
constexpr int kRingTilesBytes = (kRingFineStages + 1) * kRingFineStageBytes;           // per warp: the ring, then K and V tile of the next bucket
constexpr int kRingFoldBytes = 4 * 64 * (int) sizeof(float);                           // dpk, dpv, dpk2, dpv2 rows of a bucket
constexpr int kRingStatBytes = 2 * kBS * (int) sizeof(float);                          // lse, delta of a query block
constexpr int kRingWarpBytes = kRingTilesBytes + 2 * kRingFoldBytes + kRingFineStages * kRingStatBytes;
constexpr int kRingWindow = 64;                 // nominal entries per window: the unit whose cut buckets meet in the `partial` scratch

struct FineMaps {
  CUtensorMap q, d_o, k, v;    // [B,H,N,64] 4-D, box 16 rows
};

// SPANS: the entries of all heads, one head behind the other, in n equal pieces; the piece that holds entry p.
__host__ __device__ __forceinline__ int64_t span_begin(int64_t i, int64_t n, int64_t total) { return total * i / n; }
__device__ __forceinline__ int span_of(int64_t p, int64_t n, int64_t total) { return (int) (((p + 1) * n + total - 1) / total - 1); }

// Pooling-backward fold and scale for the ldmatrix accumulator layout: afterwards dk / dv hold the final fp32 values.  The gradient rows
// [dpk | dpv | dpk2 | dpv2] x 64 fp32 of the bucket lie at `fold`; a lane first combines four channels of one tensor in place.
template <int U>
__device__ __forceinline__ void fold_tile(const AttnP<bf16>& a, uint32_t sa, float (&dk)[8][4], float (&dv)[8][4]) {
  if constexpr (U < 8) {
    const float2 ek = lds64f<32 * U>(sa), ev = lds64f<32 * U + 256>(sa);
    dk[U][0] = fmaf(dk[U][0], a.scale, ek.x); dk[U][1] = fmaf(dk[U][1], a.scale, ek.y);
    dk[U][2] = fmaf(dk[U][2], a.scale, ek.x); dk[U][3] = fmaf(dk[U][3], a.scale, ek.y);
    dv[U][0] += ev.x; dv[U][1] += ev.y; dv[U][2] += ev.x; dv[U][3] += ev.y;
    fold_tile<U + 1>(a, sa, dk, dv);
  }
}
__device__ __forceinline__ void dkv_fine_fold_smem(const AttnP<bf16>& a, uint32_t fold, float (&dk)[8][4], float (&dv)[8][4], int lane) {
  if (a.fold) {
    const uint32_t sa = fold + 16 * lane;
    uint4 e;
    lds128<0>(e.x, e.y, e.z, e.w, sa);
    float x[4] = {__uint_as_float(e.x), __uint_as_float(e.y), __uint_as_float(e.z), __uint_as_float(e.w)};
    if (a.two_level) {
      uint4 f;
      lds128<512>(f.x, f.y, f.z, f.w, sa);
      x[0] += __uint_as_float(f.x) * (1.f / kBS); x[1] += __uint_as_float(f.y) * (1.f / kBS);
      x[2] += __uint_as_float(f.z) * (1.f / kBS); x[3] += __uint_as_float(f.w) * (1.f / kBS);
    }
    __syncwarp();
    sts128<0>(sa, make_uint4(__float_as_uint(x[0] * (1.f / kBS)), __float_as_uint(x[1] * (1.f / kBS)), __float_as_uint(x[2] * (1.f / kBS)),
                             __float_as_uint(x[3] * (1.f / kBS))));
    __syncwarp();
    fold_tile<0>(a, fold + 8 * (lane & 3), dk, dv);
  } else {
#pragma unroll
    for (int u = 0; u < 8; ++u) { dk[u][0] *= a.scale; dk[u][1] *= a.scale; dk[u][2] *= a.scale; dk[u][3] *= a.scale; }
  }
}

// Store of a finished tile through a free ring stage (`so` bytes into the ring): stmatrix writes the bf16 tile in the ring's swizzled row
// layout (the ldmatrix addresses sa_m), every lane reads back four 16-byte chunks per tensor (sa_cp: rows (lane/8) + {0, 4, 8, 12}) and
// eight lanes write one whole 128-byte row: full sectors, 8 store instructions instead of 32.
__device__ __forceinline__ void dkv_fine_store_staged(const AttnP<bf16>& a, int64_t b, int64_t h, int64_t j, float (&dk)[8][4],
                                                      float (&dv)[8][4], uint32_t sa_m, uint32_t sa_cp, uint32_t so,
                                                      uint32_t fold, int lane) {
  constexpr int TB = kRingTileBytes;
  dkv_fine_fold_smem(a, fold, dk, dv, lane);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    stsm_x4<0>((sa_m ^ (c << 5)) + so, pack_bf16(dk[2 * c][0], dk[2 * c][1]), pack_bf16(dk[2 * c][2], dk[2 * c][3]),
               pack_bf16(dk[2 * c + 1][0], dk[2 * c + 1][1]), pack_bf16(dk[2 * c + 1][2], dk[2 * c + 1][3]));
    stsm_x4<TB>((sa_m ^ (c << 5)) + so, pack_bf16(dv[2 * c][0], dv[2 * c][1]), pack_bf16(dv[2 * c][2], dv[2 * c][3]),
                pack_bf16(dv[2 * c + 1][0], dv[2 * c + 1][1]), pack_bf16(dv[2 * c + 1][2], dv[2 * c + 1][3]));
  }
  __syncwarp();
  const uint32_t sa_cp0 = sa_cp + so, sa_cp1 = (sa_cp ^ 64) + so;
  bf16* kp = a.dk.row(b, h, j * kBS + (lane >> 3)) + (lane & 7) * 8;
  bf16* vp = a.dv.row(b, h, j * kBS + (lane >> 3)) + (lane & 7) * 8;
  const int64_t ks = 4 * a.dk.sn, vs = 4 * a.dv.sn;
  uint4 x;
  lds128<0>(x.x, x.y, x.z, x.w, sa_cp0);         *reinterpret_cast<uint4*>(kp) = x;
  lds128<512>(x.x, x.y, x.z, x.w, sa_cp1);       *reinterpret_cast<uint4*>(kp + ks) = x;
  lds128<1024>(x.x, x.y, x.z, x.w, sa_cp0);      *reinterpret_cast<uint4*>(kp + 2 * ks) = x;
  lds128<1536>(x.x, x.y, x.z, x.w, sa_cp1);      *reinterpret_cast<uint4*>(kp + 3 * ks) = x;
  lds128<TB>(x.x, x.y, x.z, x.w, sa_cp0);        *reinterpret_cast<uint4*>(vp) = x;
  lds128<TB + 512>(x.x, x.y, x.z, x.w, sa_cp1);  *reinterpret_cast<uint4*>(vp + vs) = x;
  lds128<TB + 1024>(x.x, x.y, x.z, x.w, sa_cp0); *reinterpret_cast<uint4*>(vp + 2 * vs) = x;
  lds128<TB + 1536>(x.x, x.y, x.z, x.w, sa_cp1); *reinterpret_cast<uint4*>(vp + 3 * vs) = x;
  __syncwarp();
  tc::fence_async_smem();                 // the stage is refilled by the asynchronous proxy
}

// SPANS: n_pieces = spans, n_total = entries of all heads; otherwise n_pieces = windows per head, n_total = windows of all heads.
template <bool SPANS>
__global__ void __launch_bounds__(kRingWarps * 32, 1)
attn_dkv_fine_ring_kernel(AttnP<bf16> a, const __grid_constant__ FineMaps maps, float* __restrict__ partial, int n_pieces, int64_t n_total) {
  constexpr int NW = kRingWarps;
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t s_full[NW][kRingFineStages + 1];       // the ring's stages, then the next bucket's K / V
  __shared__ tc::WaitCtl s_ctl;
  __shared__ int s_next;
  // swizzled tiles: 1024-byte aligned
  unsigned char* smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  volatile tc::WaitCtl* ctl = &s_ctl;
  if (threadIdx.x == 0) {
    s_ctl.abort = 0;
    s_ctl.limit = a.wait_limit > 0 ? a.wait_limit : tc::kWaitPolls;
    s_next = 0;
  }
  if (threadIdx.x < NW * (kRingFineStages + 1)) tc::mbar_init(&s_full[0][0] + threadIdx.x, 1);
  tc::fence_mbar_init();
  pdl_wait();
  pdl_trigger();            // behind the wait: the finish kernel's first CTAs rely on the kernels in front of this one
  __syncthreads();

  const int E = (int) (a.nq1 * a.topk), n1 = (int) a.n1;
  const int R = (E + a.range_entries - 1) / a.range_entries;
  // Per-lane shared addresses of stage 0 (tiles are 1024-byte aligned, so the chunk index of an address is its bits 4..6 and a swizzle
  // partner is one XOR away):
  //   sa_cp  16-byte chunk lane % 8 of tile rows lane / 8 and lane / 8 + 8 (^ 64: + 4, + 12)
  //   sa_f   chunk 2t of row g (^ 16: chunk 2t + 1; row g + 8 is 1024 bytes on)
  //   sa_m   ldmatrix.trans row address for output channels 0..15 (^ 32 c: 16c..16c+15)
  const uint32_t ring_sa = tc::smem_u32(smem + warp * kRingTilesBytes);
  const uint32_t fold_sa = tc::smem_u32(smem + NW * kRingTilesBytes + warp * 2 * kRingFoldBytes);
  const uint32_t stat_sa = tc::smem_u32(smem + NW * (kRingTilesBytes + 2 * kRingFoldBytes) + warp * kRingFineStages * kRingStatBytes);
  const uint32_t sa_cp = ring_sa + (lane >> 3) * 128 + (((lane & 7) ^ (lane >> 3)) << 4);
  const uint32_t sa_f = ring_sa + g * 128 + (((2 * t) ^ g) << 4);
  const uint32_t sa_m = ring_sa + ((lane & 7) + ((lane >> 3) & 1) * 8) * 128 + (((lane >> 4) ^ (lane & 7)) << 4);
  const float sl2 = a.scale * kLog2e;
  float dk[8][4], dv[8][4];
  RowFrag klo, khi, vlo, vhi;               // K and V of the bucket at hand, as A operands
  int st = 0, ph = 0;                       // ring stage of the entry at hand, parity of its fill
  int kvph = 0, fold_buf = 0;               // parity of the next K / V fill, fold buffer of the bucket at hand
  // entries the CSR really holds: fewer than E when the transpose dropped out-of-range indices; ranges and offsets handed in
  // by a caller are not trusted further than these clamps and the bounds on the bucket walk below
  // SPANS: the warp's own, a head at a time.  Otherwise the warps of a CTA draw one range after another; a range that begins inside a bucket is
  // left to the warp that has the range in front of it, unless it opens a window.
  const int span = warp * (int) gridDim.x + (int) blockIdx.x;
  int bh = 0, rb = 0, left = 0;              // SPANS: head and first entry of the next piece, entries left of the span
  if (SPANS && span < n_pieces) {
    const int64_t f = span_begin(span, n_pieces, n_total);
    left = (int) (span_begin(span + 1, n_pieces, n_total) - f);
    bh = (int) (f / E) - 1;
    rb = (int) (f - (int64_t) (bh + 1) * E);
  }
  bool ok = true;
  while (ok) {
    int re, r0;                              // entries [rb, re) of head bh; the range that rb is looked up by
    if constexpr (SPANS) {
      if (left <= 0) break;
      ++bh;
      re = min(E, rb + left);
      left -= re - rb;
      r0 = rb / a.range_entries;
    } else {
      int k = 0;
      if (lane == 0) k = atomicAdd(&s_next, 1);
      k = __shfl_sync(0xffffffffu, k, 0);
      const int64_t u = blockIdx.x + (int64_t) (k >> 1) * gridDim.x;        // both ranges of a window: a left-over range is work for its neighbour
      if (u >= n_total) break;
      bh = (int) (u / n_pieces);
      r0 = (int) (u % n_pieces) * 2 + (k & 1);
      if (r0 >= R) continue;
    }
    // What the walk starts from is two rounds of loads away, each in flight at once: the ranges from r0 on and the entries in use; then the bucket
    // ends from the range's bucket on, the query blocks of the first entries, and where the bucket of the window's second range begins.  (One after the
    // other, seven rounds: l1, B=2 H=4 N=16384 60.3 us instead of 59.2, l2, B=3 H=5 N=5376 43.7 / 43.0, B=4 H=6 N=16384 152.6 / 151.5.)
    const int32_t* fl = a.flat + (int64_t) bh * E;
    int cur_qb = 0, nx_qb = 0;               // lane i: query block of entry 32 c + i of the chunk c being requested and of the one after it
    auto first_entries = [&] { if (rb + lane < E) nx_qb = __ldcg(fl + rb + lane); };
    if (SPANS) first_entries();
    const int2 rr = __ldcg(&a.ranges[(int64_t) bh * R + min(r0 + min(lane, 2), R - 1)]);
    const int E_used = (int) min((int64_t) E, max((int64_t) 0, csr_off(a, bh, n1)));
    auto bucket_of = [&](int i) { return min(max(__shfl_sync(0xffffffffu, rr.y, i), 0), n1 - 1); };
    // Bucket walk: lane l holds the end of bucket jb + l, so the bucket of an entry is the number of ends at or below it, and the next
    // non-empty bucket is known without a load while the one at hand is being worked on.
    auto bucket_end = [&](int j0) { return j0 + 1 + lane <= n1 ? (int) csr_off(a, bh, j0 + 1 + lane) : 0x7fffffff; };
    int jb = bucket_of(0), ends = bucket_end(jb), ends2 = bucket_end(jb + 32);
    const int begin_jb = (int) csr_off(a, bh, jb);
    if constexpr (SPANS) {
      re = min(re, E_used);
    } else {
      // a cut: the range's entry, or the entries' end
      auto cut = [&](int i) { return r0 + i < R ? min(max(__shfl_sync(0xffffffffu, rr.x, i), 0), E_used) : E_used; };
      const int odd = r0 & 1, x1 = __shfl_sync(0xffffffffu, rr.x, 1 - odd), begin1 = (int) csr_off(a, bh, bucket_of(1 - odd));
      rb = cut(0);
      first_entries();
      const int re1 = cut(1), re2 = cut(2);
      const bool both = (odd || r0 + 1 < R) && begin1 < x1;      // the window's second range begins inside a bucket
      if (odd && both) continue;
      re = max(both ? re2 : re1, rb);
    }
    if (rb >= re) {
      if (SPANS) rb = 0;
      continue;
    }
    const int b = bh / (int) a.H, h = bh % (int) a.H;
    // the span's or the window's head and tail slots
    float* const pieces = partial + (SPANS ? (int64_t) span : (int64_t) bh * n_pieces + r0 / (kRingWindow / kRangeEntries)) * 2 * (int64_t) kTileFloats;
    const int n = re - rb;
    auto fetch = [&](int i0) {
      if (i0 + lane < n) nx_qb = __ldcg(fl + rb + i0 + lane);
    };
    int rst = st;                            // ring stage of the next request
    const float* stat = (lane < 16 ? a.lse : a.delta) + bh * a.Nq + (lane & 15);
    auto request = [&](int i) {              // Q and dO tile by TMA, lse and delta by one 4-byte copy per lane
      if (i < n) {
        if ((i & 31) == 0) {
          cur_qb = min(max(nx_qb, 0), (int) a.nq1 - 1);      // nothing is read outside the tensors
          fetch(i + 32);
        }
        const int qb = __shfl_sync(0xffffffffu, cur_qb, i & 31);
        load_tiles_w(ring_sa + rst * kRingFineStageBytes, &maps.q, &maps.d_o, &s_full[warp][rst], kRingFineStageBytes, qb * kBS, (int) h, (int) b);
        cp_async4_sa(stat_sa + rst * kRingStatBytes + 4 * lane, stat + qb * kBS);
        rst = rst == kRingFineStages - 1 ? 0 : rst + 1;
      }
      cp_async_commit();
    };
    request(0);
    request(1);
    int j = -1, nxt = rb, j2 = 0, nxt2 = 0;  // the bucket at hand and its end, the one after it and its end
    auto find_bucket = [&](int e) {          // j2, nxt2: the bucket of entry e
      int c = __popc(__ballot_sync(0xffffffffu, ends <= e));
      while (c == 32) {
        jb += 32;
        ends = ends2;
        ends2 = bucket_end(jb + 32);
        c = __popc(__ballot_sync(0xffffffffu, ends <= e));
      }
      j2 = min(jb + c, n1 - 1);
      nxt2 = max(__shfl_sync(0xffffffffu, ends, c), e + 1);      // whatever the offsets hold, the walk moves on
    };
    // K and V tile and the pooled-gradient rows the bucket's store folds in
    auto request_bucket = [&]() {
      uint64_t* bar = &s_full[warp][kRingFineStages];
      const int rows = a.fold ? (a.two_level ? 4 : 2) : 0;
      load_tiles_w(ring_sa + kRingFineStages * kRingFineStageBytes, &maps.k, &maps.v, bar, kRingFineStageBytes + rows * 256, j2 * kBS, (int) h, (int) b);
      if (a.fold) {
        const uint32_t dst = fold_sa + (fold_buf ^ 1) * kRingFoldBytes;
        const int64_t o1 = (bh * a.n1 + j2) * kD, o2 = (bh * a.n2 + j2 / kBS) * kD;
        load_row_w(dst, a.dpk + o1, bar);
        load_row_w(dst + 256, a.dpv + o1, bar);
        if (a.two_level) {
          load_row_w(dst + 512, a.dpk2 + o2, bar);
          load_row_w(dst + 768, a.dpv2 + o2, bar);
        }
      }
    };
    const int c0 = __popc(__ballot_sync(0xffffffffu, ends <= rb)), end_c0 = __shfl_sync(0xffffffffu, ends, (c0 - 1) & 31);
    find_bucket(rb);
    bool began_before = (c0 == 0 ? begin_jb : c0 < 32 ? end_c0 : (int) csr_off(a, bh, j2)) < rb;      // the first bucket's begin lies in front of rb
    request_bucket();
    for (int i = 0; i < n; ++i) {
      const int e = rb + i;
      const uint32_t so = st * kRingFineStageBytes;
      if (!(ok = tc::warp_wait(&s_full[warp][st], ph, ctl))) break;
      cp_async_wait_group<1>();
      __syncwarp();
      const bool fresh = e >= nxt;
      if (fresh) {                                    // next non-empty bucket; the stage read an entry ago stages the store
        if (j >= 0) {
          if (!began_before) {
            dkv_fine_store_staged(a, b, h, j, dk, dv, sa_m, sa_cp, rst * kRingFineStageBytes, fold_sa + fold_buf * kRingFoldBytes, lane);
          } else {                                    // began in an earlier span
            tile_to_mem(pieces, dk, dv, lane);
          }
          began_before = false;
        }
        j = j2; nxt = nxt2;
        fold_buf ^= 1;
        if (!(ok = tc::warp_wait(&s_full[warp][kRingFineStages], kvph, ctl))) break;
        kvph ^= 1;
        constexpr int KV = kRingFineStages * kRingFineStageBytes, TB = kRingTileBytes;
        rowfrag_sa<KV>(klo, sa_f, sa_f ^ 16);
        rowfrag_sa<KV + 1024>(khi, sa_f, sa_f ^ 16);
        rowfrag_sa<KV + TB>(vlo, sa_f, sa_f ^ 16);
        rowfrag_sa<KV + TB + 1024>(vhi, sa_f, sa_f ^ 16);
        tile_zero(dk, dv);
      }
      // S^T = K.Q^T and dP^T = V.dO^T: rows = keys g, g + 8, columns = queries 2t, 2t + 1 (s0, e0) and 8 more (s1, e1)
      float s0[4], s1[4], e0[4], e1[4];
      const uint32_t f0 = sa_f + so, f1 = f0 ^ 16, m0 = sa_m + so;
      half_rows_x_keys<0, true>(s0, s1, klo, khi, f0);
      half_rows_x_keys<kRingTileBytes, true>(e0, e1, vlo, vhi, f0);
      half_rows_x_keys<0, false>(s0, s1, klo, khi, f1);
      half_rows_x_keys<kRingTileBytes, false>(e0, e1, vlo, vhi, f1);
      // The stage read an entry ago is free: its operands were consumed by products already issued.  A request keeps its warp some 270 cycles, which
      // pass beside the products above; spans, whose tiles come from L2, can wait until the exponentials are on their way too.  us, in front of the products
      // / here / behind the exponentials: spans at one level, B=4 H=6 N=4096 47.9 / 47.4 / 45.4; windows at two levels, B=1 H=5 N=40960, top-16
      // 132.8 / 130.5 / 132.0, B=8 H=6 N=16384 245.3 / 244.0 / 245.5.
      if constexpr (!SPANS) request(i + kRingFineStages - 1);
      const uint32_t sa_s = stat_sa + st * kRingStatBytes + 8 * t;
      auto half = [&](const float2 l, const float2 d, const float (&s)[4], const float (&p)[4], uint32_t& P0, uint32_t& P1, uint32_t& D0, uint32_t& D1) {
        const F2 nl = f2_mul(f2(l.x, l.y), f2(-kLog2e, -kLog2e)), nd = f2(-d.x, -d.y), sc = f2(sl2, sl2);
        float x0, x1, y0, y1;
        f2_get(f2_fma(f2(s[0], s[1]), sc, nl), x0, x1);
        f2_get(f2_fma(f2(s[2], s[3]), sc, nl), y0, y1);
        x0 = fast_exp2(x0); x1 = fast_exp2(x1); y0 = fast_exp2(y0); y1 = fast_exp2(y1);
        P0 = pack_bf16(x0, x1);
        P1 = pack_bf16(y0, y1);
        f2_get(f2_mul(f2(x0, x1), f2_add(f2(p[0], p[1]), nd)), x0, x1);
        f2_get(f2_mul(f2(y0, y1), f2_add(f2(p[2], p[3]), nd)), y0, y1);
        D0 = pack_bf16(x0, x1);
        D1 = pack_bf16(y0, y1);
      };
      uint4 P, D;                                     // P^T and dS^T / scale as A operands
      half(lds64f<0>(sa_s), lds64f<64>(sa_s), s0, e0, P.x, P.y, D.x, D.y);
      half(lds64f<32>(sa_s), lds64f<96>(sa_s), s1, e1, P.z, P.w, D.z, D.w);
      if constexpr (SPANS) request(i + kRingFineStages - 1);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t bd[4];
        ldsm_x4_trans<kRingTileBytes>(bd[0], bd[1], bd[2], bd[3], m0 ^ (c << 5));
        mma_bf16_16816(dv[2 * c], P.x, P.y, P.z, P.w, bd[0], bd[1]);
        mma_bf16_16816(dv[2 * c + 1], P.x, P.y, P.z, P.w, bd[2], bd[3]);
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t bq[4];
        ldsm_x4_trans<0>(bq[0], bq[1], bq[2], bq[3], m0 ^ (c << 5));
        mma_bf16_16816(dk[2 * c], D.x, D.y, D.z, D.w, bq[0], bq[1]);
        mma_bf16_16816(dk[2 * c + 1], D.x, D.y, D.z, D.w, bq[2], bq[3]);
      }
      if (fresh && nxt < re) {                        // K and V have been consumed: the next bucket's may overwrite them
        find_bucket(nxt);
        request_bucket();
      }
      if (st == kRingFineStages - 1) { st = 0; ph ^= 1; } else { ++st; }
    }
    if (!ok) break;
    __syncwarp();
    // the last bucket of the span; the ring is idle by now
    if (!began_before && nxt <= re) {
      dkv_fine_store_staged(a, b, h, j, dk, dv, sa_m, sa_cp, 0, fold_sa + fold_buf * kRingFoldBytes, lane);
    } else {
      tile_to_mem(pieces + (began_before ? 0 : kTileFloats), dk, dv, lane);     // reaches back or across, or continues in the next
    }
    if (SPANS) rb = 0;                       // what is left is the next head's
  }
  if (!ok) tc::abort_drain();
  __syncthreads();
  if (threadIdx.x == 0 && s_ctl.abort && a.status) atomicOr(a.status, (int) LLSA_DEV_WAIT_EXPIRED);
}

// KV blocks nobody selected: their dk / dv are the pooling-backward term alone, one row sixteen times.  A warp looks at four blocks, one per
// lane, and writes the empty ones two at a time: lane (tensor, row parity, 16-byte chunk) has both blocks' gradient rows in flight.
constexpr int kPlainPerWarp = 4;
__device__ __forceinline__ void dkv_store_unselected(const AttnP<bf16>& a, int64_t b, int64_t h, int64_t bh, int first, int lane) {
  const int n1 = (int) a.n1, jl = min(first + lane, n1 - 1);
  unsigned todo = __ballot_sync(0xffffffffu, lane < kPlainPerWarp && first + lane < n1 && csr_off(a, bh, jl + 1) <= csr_off(a, bh, jl));
  const int ten = lane >> 4, rr = (lane >> 3) & 1, c = (lane & 7) * 8;
  const View<bf16> out = ten ? a.dv : a.dk;
  const float *g1 = ten ? a.dpv : a.dpk, *g2 = ten ? a.dpv2 : a.dpk2;
  while (todo) {
    float4 e[2][2], f[2][2];
    int j[2];
    unsigned m = todo;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      j[u] = m ? first + __ffs((int) m) - 1 : -1;
      m &= m - 1;
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        e[u][v] = f[u][v] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j[u] >= 0 && a.fold) {
          e[u][v] = __ldcg(reinterpret_cast<const float4*>(g1 + (bh * a.n1 + j[u]) * kD + c + 4 * v));
          if (a.two_level) f[u][v] = __ldcg(reinterpret_cast<const float4*>(g2 + (bh * a.n2 + j[u] / kBS) * kD + c + 4 * v));
        }
      }
    }
    todo = m;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (j[u] < 0) break;
      uint32_t w[4];
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        const float4 x = e[u][v], y = f[u][v];
        const float s = 1.f / kBS;
        w[2 * v] = pack_bf16((x.x + y.x * s) * s, (x.y + y.y * s) * s);
        w[2 * v + 1] = pack_bf16((x.z + y.z * s) * s, (x.w + y.w * s) * s);
      }
      bf16* p = out.row(b, h, (int64_t) j[u] * kBS + rr) + c;
#pragma unroll
      for (int i = 0; i < 8; ++i) *reinterpret_cast<uint4*>(p + 2 * i * out.sn) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

// Buckets whose pieces lie in several windows (spans) of the kernel above.  Each of them crosses a boundary, and a boundary lies in one
// bucket: one CTA per boundary looks up that bucket (the transpose kernel left it beside the range that starts there, or in front), leaves unless
// this is the first boundary the bucket crosses, and adds the pieces in order: the tail of the window the bucket begins in, then
// the heads.  A warp owns 32 channels of one tensor, so a piece is four 128-bit loads per lane, four pieces in flight.
// The first n_plain * BH CTAs: the unselected blocks, 16 per CTA -- stores at the memory's rate next to the latency of the lookups (as extra
// CTAs or extra work of the kernel above they cost twice as much: one CTA of it fills an SM).
// Launched behind the kernel above it takes 42 us at 48 slices of 16384 tokens and 114 at 6 of 262144 (ncu, cold cache); one warp for eight buckets, looking for
// both kinds, took half as long again and twice as long.
// It is launched while the kernel above ends: the unselected blocks and the lookups need nothing of it (its CTAs let this launch begin once they have
// waited for the kernels in front of them) and take the SMs that its ragged end leaves idle; what adds pieces waits.  Whole layer, launched behind / into
// the end: one level, B=4 H=6 N=4096 189.2 / 186.5 us, B=2 H=4 N=16384 334 / 329; two levels, B=3 H=5 N=5376 164.9 / 160.1, H=5 N=40960 top-16
// 548 / 542, B=4 H=6 N=16384 641 / 634.
// What it still takes behind the end (in a graph, 24 us at 48 slices of 16384 tokens, 55 % of whose blocks are unselected, 90 at 6 of 262144, 87 %) is the memory's time
// for 4 KB a block.  No gain from: the unselected blocks written by warps of the kernel above that have run out of ranges (that kernel grows by what this one
// loses: 506 and 516 us for both at 262144); one wave of CTAs that go from boundary to boundary with the next lookups under way (50 instead of 42 us at B=1 H=5
// N=40960 top-16); eight to thirty-two blocks a warp.
__global__ void __launch_bounds__(128) attn_dkv_finish_kernel(AttnP<bf16> a, const float* __restrict__ partial, unsigned n_plain, unsigned BH, int n_spans) {
  if (blockIdx.x < n_plain * BH) {
    const int bh = (int) (blockIdx.x / n_plain), first = ((int) (blockIdx.x % n_plain) * 4 + (int) (threadIdx.x >> 5)) * kPlainPerWarp;
    dkv_store_unselected(a, bh / a.H, bh % a.H, bh, first, threadIdx.x & 31);
    if (blockIdx.x == n_plain * BH - 1) pdl_wait();      // whatever else there is, this kernel does not end before the one in front of it
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, n1 = (int) a.n1;
  const int E = (int) (a.nq1 * a.topk), range = a.range_entries, R = (E + range - 1) / range;
  const unsigned boundary = blockIdx.x - n_plain * BH;
  // offsets are clamped to [0, E] and to each other: a malformed CSR cannot send the arithmetic below outside `partial`
  int64_t bh;
  int j, c_first, c_last;
  if (n_spans > 0) {
    const int64_t total = (int64_t) BH * E, f = span_begin(boundary + 1, n_spans, total);
    bh = f / E;
    const int e = (int) (f - bh * E);
    if (e == 0) return;
    int j0 = min(max(__ldcg(&a.ranges[bh * R + e / range].y), 0), n1 - 1), c;      // its bucket begins at or in front of e
    while ((c = __popc(__ballot_sync(0xffffffffu, j0 + 1 + lane <= n1 && (int) csr_off(a, bh, j0 + 1 + lane) <= e))) == 32) j0 += 32;
    j = min(j0 + c, n1 - 1);
    const int bo = (int) min((int64_t) E, max((int64_t) 0, csr_off(a, bh, j))), be = (int) min((int64_t) E, max((int64_t) bo, csr_off(a, bh, j + 1)));
    if (bo >= e || be <= e) return;
    c_first = span_of(bh * E + bo, n_spans, total);
    if (c_first != (int) boundary) return;
    c_last = min(span_of(bh * E + be - 1, n_spans, total), n_spans - 1);
    partial += (int64_t) c_first * 2 * kTileFloats;
  } else {
    const int window = kRingWindow, n_windows = (E + window - 1) / window, at = (int) (boundary % (n_windows - 1)), edge = (at + 1) * window;
    bh = boundary / (n_windows - 1);
    j = min(max(__ldcg(&a.ranges[bh * R + edge / range].y), 0), n1 - 1);
    const int bo = (int) min((int64_t) E, max((int64_t) 0, csr_off(a, bh, j))), be = (int) min((int64_t) E, max((int64_t) bo, csr_off(a, bh, j + 1)));
    if (be - bo <= range || bo >= edge || be <= edge || bo / window != at) return;
    c_first = bo / window;
    c_last = min((be - 1) / window, n_windows - 1);
    partial += (bh * n_windows + c_first) * 2 * (int64_t) kTileFloats;
  }
  const int64_t b = bh / a.H, h = bh % a.H;
  c_last -= c_first;                                                   // pieces behind the first one
  pdl_wait();                                                          // for the pieces
  const int ten = warp >> 1, u0 = (warp & 1) * 4;                      // tiles u0 .. u0 + 3 of dk / dv: tile u holds channels 8u + 2t, +1 of rows g, g + 8
  float acc[4][4];
#pragma unroll
  for (int u = 0; u < 4; ++u) acc[u][0] = acc[u][1] = acc[u][2] = acc[u][3] = 0.f;
  for (int c0 = 0; c0 <= c_last; c0 += 4) {
    float4 x[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = min(c0 + i, c_last);
      const float4* p = reinterpret_cast<const float4*>(partial + (c * 2 + (c == 0 ? 1 : 0)) * (int64_t) kTileFloats) + (8 * ten + u0) * 32 + lane;
#pragma unroll
      for (int u = 0; u < 4; ++u) x[i][u] = __ldcg(p + u * 32);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (c0 + i > c_last) break;
#pragma unroll
      for (int u = 0; u < 4; ++u) { acc[u][0] += x[i][u].x; acc[u][1] += x[i][u].y; acc[u][2] += x[i][u].z; acc[u][3] += x[i][u].w; }
    }
  }
  const float *g1 = (ten ? a.dpv : a.dpk) + (bh * a.n1 + j) * kD, *g2 = a.two_level ? (ten ? a.dpv2 : a.dpk2) + (bh * a.n2 + j / kBS) * kD : nullptr;
  const View<bf16> out = ten ? a.dv : a.dk;
  const float mul = ten ? 1.f : a.scale;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int c = 8 * (u0 + u) + 2 * t;
    float2 e = make_float2(0.f, 0.f);
    if (a.fold) {
      e = __ldcg(reinterpret_cast<const float2*>(g1 + c));
      if (a.two_level) {
        const float2 f = __ldcg(reinterpret_cast<const float2*>(g2 + c));
        e.x += f.x * (1.f / kBS); e.y += f.y * (1.f / kBS);
      }
    }
    *reinterpret_cast<uint32_t*>(out.row(b, h, (int64_t) j * kBS + g) + c) = pack_bf16(acc[u][0] * mul + e.x * (1.f / kBS), acc[u][1] * mul + e.y * (1.f / kBS));
    *reinterpret_cast<uint32_t*>(out.row(b, h, (int64_t) j * kBS + g + 8) + c) = pack_bf16(acc[u][2] * mul + e.x * (1.f / kBS), acc[u][3] * mul + e.y * (1.f / kBS));
  }
}

int zero_pooled_acc(const LlsaAttnArgs* g, cudaStream_t st);

int launch_attn_bwd_mma(const LlsaAttnArgs* g, cudaStream_t st) {
  if (!mma_path_ok(g, true)) {
    note_scalar_path();
    return launch_attn_bwd_generic(g, st);
  }
  AttnP<bf16> a = build_attn_params<bf16>(g, true);
  const unsigned BH = (unsigned) (g->q->shape[0] * a.H);
  const int mask = g->stage_mask ? g->stage_mask : 7;
  // pooled keys on tcgen05 (attn_pooled_bwd_tc.cu): the dQ kernel then covers the fine blocks only and the
  // tensor-core kernel adds the pooled part of dq and produces the pooled-key gradients
  const bool tc = pooled_bwd_tc_ok(a) && !g->no_tcgen05;
  // other pooled key lists: the key-loop tcgen05 kernels (dQ, then the key-major dK/dV); a list whose fine part of dq has to cross with its
  // remainder takes dq in one kernel if the caller gave no room for that
  const bool rem = remainder_wanted(a, true);
  if (!rem) a.rem = nullptr;
  const bool loop_dkv = !tc && pooled_dq_loop_tc_keys(a) > 0 && !g->no_tcgen05, loop_dq = loop_dkv && (!rem || a.rem);
  if (mask & 1) {
    constexpr int NWQ = 4;
    AttnP<bf16> aq = a;
    if (tc || loop_dq) aq.p1_blocks = aq.p2_blocks = 0;
    const int n_all = aq.p1_blocks + aq.p2_blocks;
    // The fine kernel clears the pooled-gradient accumulators itself: a memset beside it (on another stream) finds no room until its last wave and holds up
    // the stage that follows
    const bool zero = !(g->stage_mask & 8);
    if (zero && n_all) {
      int rc = zero_pooled_acc(g, st);
      if (rc) return rc;
    }
    const int n_smem = n_all < 12 ? n_all : 12;   // 12 tiles = 54 KB of K+V, three CTAs per SM
    const size_t smem = (size_t) n_smem * kBS * kSmemPitch * sizeof(bf16) * 2;
    if (n_all == 0) {
      KvMaps maps;
      memset(&maps, 0, sizeof(maps));
      int rc;
      if ((rc = tma::make_map_bhnd(&maps.k, g->k, kBS))) return rc;
      if ((rc = tma::make_map_bhnd(&maps.v, g->v, kBS))) return rc;
      const size_t ring = (size_t) NWQ * kDqStages * 2 * kRingTileBytes + 1024;
      auto fine = loop_dq && a.rem ? attn_dq_fine_kernel<NWQ, true> : attn_dq_fine_kernel<NWQ, false>;
      LLSA_SMEM_LIMIT(fine, ring);
      launch_pdl(fine, dim3((unsigned) (a.nq1 / NWQ), BH), NWQ * 32, ring, st, aq, maps, zero);
      LLSA_LAUNCH_OK("attn_dq_fine_kernel");
    } else {
      LLSA_SMEM_LIMIT((attn_dq_mma_kernel<NWQ>), smem);
      attn_dq_mma_kernel<NWQ><<<dim3((unsigned) (a.nq1 / NWQ), BH), NWQ * 32, smem, st>>>(aq, n_smem);
      LLSA_LAUNCH_OK("attn_dq_mma_kernel");
    }
  }
  if ((mask & 2) && tc) {
    int rc = launch_attn_bwd_pooled_tc(g, a, BH, st);
    if (rc) return rc;
  } else if ((mask & 2) && a.p1_blocks + a.p2_blocks > 0) {
    if (loop_dq) {
      int rc = launch_attn_dq_pooled_loop_tc(g, a, BH, st);
      if (rc) return rc;
    }
    if (loop_dkv) {
      int rc = launch_attn_dkv_pooled_loop_tc(g, a, BH, st);
      if (rc) return rc;
    } else {
      constexpr int NWP = 8;
      const size_t smem = (size_t) 2 * kBS * kBS * kSmemPitch * sizeof(bf16) + 2 * kBS * kBS * sizeof(float);
      LLSA_SMEM_LIMIT((attn_dkv_pooled_kernel<NWP>), smem);
      attn_dkv_pooled_kernel<NWP><<<dim3((unsigned) (a.nq1 / kBS), BH), NWP * 32, smem, st>>>(a);
      LLSA_LAUNCH_OK("attn_dkv_pooled_kernel");
    }
  }
  if (mask & 4) {
    const int64_t E = a.nq1 * a.topk;
    const int n_windows = (int) ((E + kRingWindow - 1) / kRingWindow);
    float* partial = (float*) g->dkv_partial->ptr;
    FineMaps maps;
    memset(&maps, 0, sizeof(maps));
    int rc;
    if ((rc = tma::make_map_bhnd(&maps.q, g->q, kBS))) return rc;
    if ((rc = tma::make_map_bhnd(&maps.d_o, g->d_o, kBS))) return rc;
    if ((rc = tma::make_map_bhnd(&maps.k, g->k, kBS))) return rc;
    if ((rc = tma::make_map_bhnd(&maps.v, g->v, kBS))) return rc;
    int dev = 0, sms = 148;
    LLSA_CUDA_OK(cudaGetDevice(&dev));
    LLSA_CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const size_t ring = (size_t) kRingWarps * kRingWarpBytes + 1024;
    int n_spans = 0;
    if (a.range_entries == kRangeEntries) {
      static_assert(kRingWindow == 2 * kRangeEntries, "a window is two ranges");
      const int64_t total = (int64_t) n_windows * BH;
      LLSA_SMEM_LIMIT((attn_dkv_fine_ring_kernel<false>), ring);
      launch_pdl(attn_dkv_fine_ring_kernel<false>, dim3((unsigned) (total < sms ? total : sms)), kRingWarps * 32, ring, st, a, maps, partial, n_windows, total);
    } else {
      const int64_t total = E * BH, room = g->dkv_partial->shape[0] * g->dkv_partial->shape[1] * g->dkv_partial->shape[2] * g->dkv_partial->shape[3] / (2 * kTileFloats);
      n_spans = (int) std::min({(total + kSpanEntries - 1) / kSpanEntries, (int64_t) sms * kRingWarps, room});
      LLSA_SMEM_LIMIT((attn_dkv_fine_ring_kernel<true>), ring);
      launch_pdl(attn_dkv_fine_ring_kernel<true>, dim3((unsigned) std::min(n_spans, sms)), kRingWarps * 32, ring, st, a, maps, partial, n_spans, total);
    }
    LLSA_LAUNCH_OK("attn_dkv_fine_ring_kernel");
    const unsigned n_plain = (unsigned) ((a.n1 + 4 * kPlainPerWarp - 1) / (4 * kPlainPerWarp)), boundaries = n_spans ? (unsigned) n_spans - 1 : (unsigned) (n_windows - 1) * BH;
    launch_pdl(attn_dkv_finish_kernel, dim3(n_plain * BH + boundaries), 128, 0, st, a, (const float*) partial, n_plain, BH, n_spans);
    LLSA_LAUNCH_OK("attn_dkv_finish_kernel");
  }
  return LLSA_OK;
}

}  // namespace llsa
