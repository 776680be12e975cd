// Block-sparse LLSA forward on the tensor cores (bf16, D = 64, 16-token blocks).
// Reference: _sparse_indices_attn_res_fwd (sparse_attention_res_1.py:9-120) and
// _sparse_indices_attn_res_2_2_fwd (sparse_attention_res_2.py:9-163).
//
// attn_fwd_fine_kernel (below) takes the fine blocks where tcgen05 kernels take the pooled keys.  Otherwise -- no pooled keys at all, the
// tcgen05 kernels switched off, or a list that wants `remainder` and has none -- attn_fwd_mma_kernel takes both:
//
// One warp owns one 16-row query block (the m16 of mma.sync.m16n8k16); a CTA of
// NW warps owns NW consecutive query blocks, which always share their parent
// block and therefore the same pooled keys.
//   * Pooled key/value tiles (the children of the parent's selected level-2
//     blocks and the level-2 keys; all level-1 keys in the one-level form) are
//     copied once per CTA into shared memory with cp.async while the fine stage
//     runs, then read by every warp as conflict-free 128-bit fragments.  Tiles
//     beyond the shared-memory budget are streamed like fine blocks.
//   * Fine key/value blocks are private to a query block: they go from global
//     memory straight into mma operand registers (mma_frag.cuh) with the next
//     block's loads in flight behind the current block's math.
// The softmax runs online, one 16-key block at a time, in the exp2 domain; a
// pooled key's weight enters as +log2(weight) on its logit, which is what
// `l += l_ij * W; acc += P.V * W` in the reference amounts to.
#include <string.h>

#include <type_traits>

#include "attn.cuh"
#include "mma_frag.cuh"
#include "tc05.cuh"
#include "tma.cuh"

namespace llsa {

struct FwdState {
  float o[8][4];
  float m0, m1, l0, l1;
};

// First half of a 16-key block: S = Q.K^T and the online-softmax update; returns P (bf16) as the
// four A registers of the P.V product.  The key fragments are dead afterwards.
__device__ __forceinline__ void fwd_scores(FwdState& st, const RowFrag& qlo, const RowFrag& qhi, const RowFrag& k0, const RowFrag& k1,
                                           float sl2, float lw, uint32_t (&pa)[4]) {
  float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
  mma_rows_x_keys(s0, s1, qlo, qhi, k0, k1);
#pragma unroll
  for (int c = 0; c < 4; ++c) { s0[c] = fmaf(s0[c], sl2, lw); s1[c] = fmaf(s1[c], sl2, lw); }
  const float mn0 = fmaxf(st.m0, quad_max(fmaxf(fmaxf(s0[0], s0[1]), fmaxf(s1[0], s1[1]))));
  const float mn1 = fmaxf(st.m1, quad_max(fmaxf(fmaxf(s0[2], s0[3]), fmaxf(s1[2], s1[3]))));
  const float al0 = fast_exp2(st.m0 - mn0), al1 = fast_exp2(st.m1 - mn1);
  st.m0 = mn0; st.m1 = mn1;
  s0[0] = fast_exp2(s0[0] - mn0); s0[1] = fast_exp2(s0[1] - mn0); s1[0] = fast_exp2(s1[0] - mn0); s1[1] = fast_exp2(s1[1] - mn0);
  s0[2] = fast_exp2(s0[2] - mn1); s0[3] = fast_exp2(s0[3] - mn1); s1[2] = fast_exp2(s1[2] - mn1); s1[3] = fast_exp2(s1[3] - mn1);
  st.l0 = st.l0 * al0 + (s0[0] + s0[1] + s1[0] + s1[1]);   // per-lane partial sums; reduced over the quad at the end
  st.l1 = st.l1 * al1 + (s0[2] + s0[3] + s1[2] + s1[3]);
#pragma unroll
  for (int j = 0; j < 8; ++j) { st.o[j][0] *= al0; st.o[j][1] *= al0; st.o[j][2] *= al1; st.o[j][3] *= al1; }
  // the two C tiles of S are the k16 halves of the A operand
  pa[0] = pack_bf16(s0[0], s0[1]); pa[1] = pack_bf16(s0[2], s0[3]); pa[2] = pack_bf16(s1[0], s1[1]); pa[3] = pack_bf16(s1[2], s1[3]);
}

struct GlobalBlock {
  const bf16* k;
  const bf16* v;
  int64_t ks, vs;
  float lw;
};

// Block gi of the list streamed from global memory: the fine blocks, then the pooled tiles that
// did not fit in shared memory.  gi is warp-uniform; lane i of my_fine holds fine block i.
__device__ __forceinline__ GlobalBlock global_block(const AttnP<bf16>& a, int64_t b, int64_t h, int64_t bh, int64_t qb, int gi, int my_fine,
                                                    int n_smem_tiles, float lw1, float lw2) {
  GlobalBlock r;
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

// Copies pooled tiles 0..n_tiles-1 of the query group of `qb0` into shared memory (K and V), asynchronously.
__device__ __forceinline__ void stage_pooled_tiles(const AttnP<bf16>& a, int64_t bh, int64_t qb0, int n_tiles, bf16* sk, bf16* sv) {
  for (int c = threadIdx.x; c < n_tiles * kBS * 8; c += blockDim.x) {
    const int tile = c >> 7, row = (c >> 3) & 15, ch = (c & 7) * 8;
    int64_t off;
    const bf16 *gk, *gv;
    if (tile < a.p1_blocks) {
      off = (bh * a.n1 + p1_block(a, bh, qb0, tile) * kBS + row) * kD + ch;
      gk = a.pk + off; gv = a.pv + off;
    } else {
      off = (bh * a.n2 + (int64_t) (tile - a.p1_blocks) * kBS + row) * kD + ch;
      gk = a.pk2 + off; gv = a.pv2 + off;
    }
    const int so = (tile * kBS + row) * kSmemPitch + ch;
    cp_async16(sk + so, gk);
    cp_async16(sv + so, gv);
  }
  cp_async_commit();
}

template <int NW>
__global__ void __launch_bounds__(NW * 32, 2) attn_fwd_mma_kernel(AttnP<bf16> a, int n_smem_tiles) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  bf16* sk = reinterpret_cast<bf16*>(smem_raw);
  bf16* sv = sk + n_smem_tiles * kBS * kSmemPitch;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int64_t qb0 = (int64_t) blockIdx.x * NW, qb = qb0 + warp, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
  stage_pooled_tiles(a, bh, qb0, n_smem_tiles, sk, sv);

  const int my_fine = lane < a.topk ? (int) fine_block(a, bh, qb, lane) : 0;
  const float lw1 = log2f(a.w1), lw2 = log2f(a.w2);
  const float sl2 = a.scale * 1.4426950408889634f;
  RowFrag qlo, qhi;
  load_rowfrag(qlo, a.q.row(b, h, qb * kBS + g), t);
  load_rowfrag(qhi, a.q.row(b, h, qb * kBS + g + 8), t);

  FwdState st;
#pragma unroll
  for (int j = 0; j < 8; ++j) st.o[j][0] = st.o[j][1] = st.o[j][2] = st.o[j][3] = 0.f;
  st.m0 = st.m1 = -INFINITY;
  st.l0 = st.l1 = 0.f;

  // ---- blocks streamed from global memory, next block's loads in flight behind the math
  const int n_pooled = a.p1_blocks + a.p2_blocks;
  const int n_glob = a.topk + (n_pooled - n_smem_tiles);
  {
    RowFrag k0, k1;
    ColFrag v;
    GlobalBlock r = global_block(a, b, h, bh, qb, 0, my_fine, n_smem_tiles, lw1, lw2);
    load_rowfrag(k0, r.k + (int64_t) g * r.ks, t);
    load_rowfrag(k1, r.k + (int64_t) (g + 8) * r.ks, t);
    load_colfrag(v, r.v, r.vs, g, t);
    for (int gi = 0; gi < n_glob; ++gi) {
      if (gi + 2 < n_glob) {   // two blocks ahead: K rows (lanes 0..15) and V rows (lanes 16..31) towards L1
        const GlobalBlock f = global_block(a, b, h, bh, qb, gi + 2, my_fine, n_smem_tiles, lw1, lw2);
        if (lane < 16) prefetch_tile_rows(f.k, f.ks, lane);
        else prefetch_tile_rows(f.v, f.vs, lane - 16);
      }
      uint32_t pa[4];
      fwd_scores(st, qlo, qhi, k0, k1, sl2, r.lw, pa);
      const bool more = gi + 1 < n_glob;
      if (more) {   // the key registers are free: start the next block's keys
        r = global_block(a, b, h, bh, qb, gi + 1, my_fine, n_smem_tiles, lw1, lw2);
        load_rowfrag(k0, r.k + (int64_t) g * r.ks, t);
        load_rowfrag(k1, r.k + (int64_t) (g + 8) * r.ks, t);
      }
      mma_x_cols(st.o, pa[0], pa[1], pa[2], pa[3], v);
      if (more) load_colfrag(v, r.v, r.vs, g, t);
    }
  }
  // ---- pooled tiles shared by the CTA
  cp_async_wait_all();
  __syncthreads();
  for (int ip = 0; ip < n_smem_tiles; ++ip) {
    RowFrag k0, k1;
    ColFrag v;
    const bf16* tk = sk + ip * kBS * kSmemPitch;
    load_rowfrag_smem(k0, tk + g * kSmemPitch, t);
    load_rowfrag_smem(k1, tk + (g + 8) * kSmemPitch, t);
    load_colfrag_smem(v, sv + ip * kBS * kSmemPitch, g, t);
    uint32_t pa[4];
    fwd_scores(st, qlo, qhi, k0, k1, sl2, ip < a.p1_blocks ? lw1 : lw2, pa);
    mma_x_cols(st.o, pa[0], pa[1], pa[2], pa[3], v);
  }

  const float l0 = quad_sum(st.l0), l1 = quad_sum(st.l1);
  store_acc_row<0>(a.o.row(b, h, qb * kBS + g), st.o, t, 1.f / l0);
  store_acc_row<1>(a.o.row(b, h, qb * kBS + g + 8), st.o, t, 1.f / l1);
  if (t == 0) {
    a.lse[bh * a.Nq + qb * kBS + g] = (st.m0 + log2f(l0)) * 0.6931471805599453f;
    a.lse[bh * a.Nq + qb * kBS + g + 8] = (st.m1 + log2f(l1)) * 0.6931471805599453f;
  }
}

// Fine stage alone (the pooled stages then run on tcgen05, attn_pooled_tc.cu, and merge into the o / lse written here): one warp per query
// block.  The selected K / V tiles go through a per-warp ring of three stages, two tiles of one tensor each, filled by TMA two stages
// ahead (one lane issues; no address arithmetic, no shared-memory store slots).  The blocks are taken GP pairs at a time: the S tiles of a
// group first, one softmax update, then P.V with V read by ldmatrix.trans.  Four blocks a group (GP = 2) halve the updates against two;
// GP = 1 is for a top-k that is not a multiple of four.  Bound by the gather from L2, 4 KB per (query block, selected block):
// 127 us at 8 x 6 slices of 16384 tokens, top 8 (143 with cp.async rings of single tiles, every lane copying).
constexpr int kFineStages = 3;
constexpr int kFineStageBytes = 2 * kRingTileElems * (int) sizeof(bf16);
struct FineKvMaps {
  CUtensorMap k, v;            // [B,H,N,64] 4-D, box 16 rows
};

// One lane requests rows [r0, r0 + 16) and [r1, r1 + 16) of one (head, batch) as neighbouring 2 KB tiles.
__device__ __forceinline__ void load_two_tiles_w(uint32_t dst, const CUtensorMap* m, uint64_t* bar, int r0, int r1, int h, int b) {
  asm volatile(
      "{\n\t.reg .pred e;\n\t.reg .b32 d;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "add.u32 d, %0, 2048;\n\t"
      "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%2], 4096;\n\t"
      "@e cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%7, %3, %5, %6}], [%2];\n\t"
      "@e cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [d], [%1, {%7, %4, %5, %6}], [%2];\n\t"
      "}" ::"r"(dst), "l"(m), "r"(tc::smem_u32(bar)), "r"(r0), "r"(r1), "r"(h), "r"(b), "r"(0)
      : "memory");
}

// REM: what rounding o to bf16 leaves over goes to a.rem, for the pooled stage to add (remainder_wanted).
template <int NW, int GP, bool REM>
__global__ void __launch_bounds__(NW * 32, 16 / NW) attn_fwd_fine_kernel(AttnP<bf16> a, const __grid_constant__ FineKvMaps maps) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t s_full[NW][kFineStages];
  __shared__ tc::WaitCtl s_ctl[NW];             // a warp's own: the warps of a CTA share nothing
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint32_t ring_sa = ((tc::smem_u32(smem_raw) + 1023u) & ~1023u) + warp * kFineStages * kFineStageBytes;
  volatile tc::WaitCtl* ctl = &s_ctl[warp];
  if (lane < kFineStages) tc::mbar_init(&s_full[warp][lane], 1);
  if (lane == 0) {
    ctl->abort = 0;
    ctl->limit = a.wait_limit > 0 ? a.wait_limit : tc::kWaitPolls;
  }
  tc::fence_mbar_init();
  __syncwarp();
  pdl_trigger();
  pdl_wait();
  const int64_t qb = (int64_t) blockIdx.x * NW + warp, bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
  const int my_row = lane < a.topk ? (int) fine_block(a, bh, qb, lane) * kBS : 0;
  int rst = 0;
  auto request = [&](const CUtensorMap* m, int pair) {
    load_two_tiles_w(ring_sa + rst * kFineStageBytes, m, &s_full[warp][rst], __shfl_sync(0xffffffffu, my_row, 2 * pair),
                     __shfl_sync(0xffffffffu, my_row, 2 * pair + 1), (int) h, (int) b);
    rst = rst == kFineStages - 1 ? 0 : rst + 1;
  };
  // the stages come as the K pairs of a group, then its V pairs; two are requested ahead
  request(&maps.k, 0);
  if constexpr (GP == 2) request(&maps.k, 1); else request(&maps.v, 0);
  // shared addresses of stage 0: chunks 2t, 2t + 1 of row g (sa_f, sa_f ^ 16; row g + 8 is 1024 bytes on), ldmatrix rows of channels 0..15
  // (sa_m; ^ 32 c: channels 16c..)
  const uint32_t sa_f = ring_sa + g * 128 + (((2 * t) ^ g) << 4);
  const uint32_t sa_m = ring_sa + ((lane & 7) + ((lane >> 3) & 1) * 8) * 128 + (((lane >> 4) ^ (lane & 7)) << 4);
  RowFrag qlo, qhi;
  load_rowfrag(qlo, a.q.row(b, h, qb * kBS + g), t);
  load_rowfrag(qhi, a.q.row(b, h, qb * kBS + g + 8), t);
  const float sl2 = a.scale * 1.4426950408889634f;
  const F2 sl22 = f2(sl2, sl2);
  float o[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
  float m0 = -INFINITY, m1 = -INFINITY;
  F2 l0 = f2(0.f, 0.f), l1 = f2(0.f, 0.f);      // per-lane partial sums of rows g, g + 8; reduced over the quad at the end
  const int n_pairs = a.topk / 2;
  int st = 0, ph = 0;
  bool ok = true;
  auto advance = [&]() {
    if (st == kFineStages - 1) { st = 0; ph ^= 1; } else { ++st; }
  };
  for (int gp = 0; gp < n_pairs; gp += GP) {
    float sc[2 * GP][2][4];
    uint32_t pa[2 * GP][4];
#pragma unroll
    for (int p = 0; p < GP; ++p) {
      if (!(ok = tc::warp_wait(&s_full[warp][st], ph, ctl))) break;
      // into the stage read last time: its operands were consumed by products already issued
      if constexpr (GP == 2) request(&maps.v, gp + p);
      else if (gp + 1 < n_pairs) request(&maps.k, gp + 1);
      const uint32_t f0 = sa_f + st * kFineStageBytes, f1 = f0 ^ 16;
      half_rows_x_keys<0, true>(sc[2 * p][0], sc[2 * p][1], qlo, qhi, f0);
      half_rows_x_keys<2048, true>(sc[2 * p + 1][0], sc[2 * p + 1][1], qlo, qhi, f0);
      half_rows_x_keys<0, false>(sc[2 * p][0], sc[2 * p][1], qlo, qhi, f1);
      half_rows_x_keys<2048, false>(sc[2 * p + 1][0], sc[2 * p + 1][1], qlo, qhi, f1);
      advance();
    }
    if (!ok) break;
    float x0 = -INFINITY, x1 = -INFINITY;
#pragma unroll
    for (int u = 0; u < 2 * GP; ++u)
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        x0 = fmax3(x0, sc[u][n][0], sc[u][n][1]);
        x1 = fmax3(x1, sc[u][n][2], sc[u][n][3]);
      }
    const float mn0 = fmaxf(m0, quad_max(x0) * sl2), mn1 = fmaxf(m1, quad_max(x1) * sl2);
    if (gp > 0) {
      const float al0 = fast_exp2(m0 - mn0), al1 = fast_exp2(m1 - mn1);
      l0 = f2_mul(l0, f2(al0, al0)); l1 = f2_mul(l1, f2(al1, al1));
#pragma unroll
      for (int u = 0; u < 8; ++u) { o[u][0] *= al0; o[u][1] *= al0; o[u][2] *= al1; o[u][3] *= al1; }
    }
    m0 = mn0; m1 = mn1;
    const F2 nm0 = f2(-mn0, -mn0), nm1 = f2(-mn1, -mn1);
    auto probs = [&](float y0, float y1, F2 nm, F2& l) {
      f2_get(f2_fma(f2(y0, y1), sl22, nm), y0, y1);
      y0 = fast_exp2(y0); y1 = fast_exp2(y1);
      l = f2_add(l, f2(y0, y1));
      return pack_bf16(y0, y1);
    };
#pragma unroll
    for (int u = 0; u < 2 * GP; ++u) {          // the two C tiles of S are the k16 halves of the A operand
      pa[u][0] = probs(sc[u][0][0], sc[u][0][1], nm0, l0); pa[u][1] = probs(sc[u][0][2], sc[u][0][3], nm1, l1);
      pa[u][2] = probs(sc[u][1][0], sc[u][1][1], nm0, l0); pa[u][3] = probs(sc[u][1][2], sc[u][1][3], nm1, l1);
    }
#pragma unroll
    for (int p = 0; p < GP; ++p) {
      if (!(ok = tc::warp_wait(&s_full[warp][st], ph, ctl))) break;
      if (gp + GP < n_pairs) request(GP == 2 ? &maps.k : &maps.v, gp + GP + p);
      const uint32_t vm = sa_m + st * kFineStageBytes;
      auto product = [&](auto imm, const uint32_t (&w)[4]) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t r0, r1, r2, r3;
          ldsm_x4_trans<decltype(imm)::value>(r0, r1, r2, r3, vm ^ (c << 5));
          mma_bf16_16816(o[2 * c], w[0], w[1], w[2], w[3], r0, r1);
          mma_bf16_16816(o[2 * c + 1], w[0], w[1], w[2], w[3], r2, r3);
        }
      };
      product(std::integral_constant<int, 0>{}, pa[2 * p]);
      product(std::integral_constant<int, 2048>{}, pa[2 * p + 1]);
      advance();
    }
    if (!ok) break;
  }
  if (!ok) {
    if (lane < kBS) a.lse[bh * a.Nq + qb * kBS + lane] = __int_as_float(0x7fc00000);      // NaN: not completed; the pooled stage passes it on
    tc::abort_drain();
    if (lane == 0 && a.status) atomicOr(a.status, (int) LLSA_DEV_WAIT_EXPIRED);
    return;
  }
  float y0, y1, z0, z1;
  f2_get(l0, y0, y1); f2_get(l1, z0, z1);
  const float s0 = quad_sum(y0 + y1), s1 = quad_sum(z0 + z1), i0 = 1.f / s0, i1 = 1.f / s1;
  if (t == 0) {
    a.lse[bh * a.Nq + qb * kBS + g] = (m0 + log2f(s0)) * 0.6931471805599453f;
    a.lse[bh * a.Nq + qb * kBS + g + 8] = (m1 + log2f(s1)) * 0.6931471805599453f;
  }
  // accumulator tile u holds channels 8u + 2t, 8u + 2t + 1 of rows g (c0, c1) and g + 8 (c2, c3): through the idle ring to whole rows
  __syncwarp();
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    float x[2][4];
    uint32_t w[4];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      x[u][0] = o[2 * c + u][0] * i0; x[u][1] = o[2 * c + u][1] * i0; x[u][2] = o[2 * c + u][2] * i1; x[u][3] = o[2 * c + u][3] * i1;
      w[2 * u] = pack_bf16(x[u][0], x[u][1]);
      w[2 * u + 1] = pack_bf16(x[u][2], x[u][3]);
    }
    stsm_x4<0>(sa_m ^ (c << 5), w[0], w[1], w[2], w[3]);
    if (REM)
      stsm_x4<2048>(sa_m ^ (c << 5), pack_rest(x[0][0], x[0][1], w[0]), pack_rest(x[0][2], x[0][3], w[1]), pack_rest(x[1][0], x[1][1], w[2]),
                    pack_rest(x[1][2], x[1][3], w[3]));
  }
  __syncwarp();
  const uint32_t sa_cp = ring_sa + (lane >> 3) * 128 + (((lane & 7) ^ (lane >> 3)) << 4);
  bf16* op = a.o.row(b, h, qb * kBS + (lane >> 3)) + (lane & 7) * 8;
  const int64_t os = 4 * a.o.sn;
  uint4 x;
  lds128<0>(x.x, x.y, x.z, x.w, sa_cp);         *reinterpret_cast<uint4*>(op) = x;
  lds128<512>(x.x, x.y, x.z, x.w, sa_cp ^ 64);  *reinterpret_cast<uint4*>(op + os) = x;
  lds128<1024>(x.x, x.y, x.z, x.w, sa_cp);      *reinterpret_cast<uint4*>(op + 2 * os) = x;
  lds128<1536>(x.x, x.y, x.z, x.w, sa_cp ^ 64); *reinterpret_cast<uint4*>(op + 3 * os) = x;
  if (REM) {
    bf16* rp = a.rem + (bh * a.Nq + qb * kBS + (lane >> 3)) * kD + (lane & 7) * 8;
    lds128<2048>(x.x, x.y, x.z, x.w, sa_cp);             *reinterpret_cast<uint4*>(rp) = x;
    lds128<2048 + 512>(x.x, x.y, x.z, x.w, sa_cp ^ 64);  *reinterpret_cast<uint4*>(rp + 4 * kD) = x;
    lds128<2048 + 1024>(x.x, x.y, x.z, x.w, sa_cp);      *reinterpret_cast<uint4*>(rp + 8 * kD) = x;
    lds128<2048 + 1536>(x.x, x.y, x.z, x.w, sa_cp ^ 64); *reinterpret_cast<uint4*>(rp + 12 * kD) = x;
  }
}

// A bf16 call whose operands miss the tensor-core kernels' limits still runs, on the scalar kernels and many times
// slower: the call succeeds, and the thread's error string says why so that a caller who wonders can find out.
void note_scalar_path() {
  set_error("note: bf16 operands ran on the scalar kernels (the tensor-core kernels need 32-byte aligned rows, "
            "batch/head/token strides that are multiples of 16 elements and at least a row, and top-k <= 32)");
}

bool mma_path_ok(const LlsaAttnArgs* g, bool bwd) {
  if (g->topk > 32 || (g->pk2 && g->topk_p > 32)) return false;
  // 256-bit fragment loads need 32-byte aligned rows
  const LlsaTensor* ts[8] = {g->q, g->k, g->v, g->o, bwd ? g->d_o : nullptr, bwd ? g->dq : nullptr, bwd ? g->dk : nullptr, bwd ? g->dv : nullptr};
  for (const LlsaTensor* t : ts) {
    if (!t) continue;
    if ((uintptr_t) t->ptr % 32) return false;
    for (int i = 0; i < 3; ++i)
      if (t->shape[i] != 1 && (t->stride[i] % 16 || t->stride[i] < kD)) return false;      // a tensor map's strides reach past a row
  }
  return ((uintptr_t) g->pk->ptr % 32) == 0 && ((uintptr_t) g->pv->ptr % 32) == 0 &&
         (!g->pk2 || (((uintptr_t) g->pk2->ptr % 32) == 0 && ((uintptr_t) g->pv2->ptr % 32) == 0));
}

int pooled_smem_tiles(int n_pooled) { return n_pooled < 20 ? n_pooled : 20; }   // 20 tiles = 90 KB of K+V, two CTAs per SM

int launch_attn_fwd_mma(const LlsaAttnArgs* g, cudaStream_t st) {
  if (!mma_path_ok(g, false)) {
    note_scalar_path();
    return launch_attn_fwd_generic(g, st);
  }
  AttnP<bf16> a = build_attn_params<bf16>(g, false);
  constexpr int NW = 8;
  const int64_t BH = g->q->shape[0] * a.H;
  // all pooled keys of a row at once where they fit (64, 128, 192 keys), else chunk by chunk; a list whose fine part has to cross with its
  // remainder takes the one-kernel form below if the caller gave no room for that
  const bool rem = remainder_wanted(a, false);
  if (!rem) a.rem = nullptr;
  const bool loop_tc = !pooled_tc_keys(a) && pooled_loop_tc_keys(a) > 0 && (!rem || a.rem);
  if ((pooled_tc_keys(a) || loop_tc) && !g->no_tcgen05) {
    // fine blocks on mma.sync (o and lse of the fine part alone), pooled keys on tcgen05, merged there
    FineKvMaps maps;
    memset(&maps, 0, sizeof(maps));
    int rc;
    if ((rc = tma::make_map_bhnd(&maps.k, g->k, kBS))) return rc;
    if ((rc = tma::make_map_bhnd(&maps.v, g->v, kBS))) return rc;
    constexpr int NWF = 4;
    const size_t ring = (size_t) NWF * kFineStages * kFineStageBytes + 1024;
    const dim3 fine_grid((unsigned) (a.nq1 / NWF), (unsigned) BH);
    auto fine = a.topk % 4 == 0 ? (a.rem ? attn_fwd_fine_kernel<NWF, 2, true> : attn_fwd_fine_kernel<NWF, 2, false>)
                                : (a.rem ? attn_fwd_fine_kernel<NWF, 1, true> : attn_fwd_fine_kernel<NWF, 1, false>);
    LLSA_SMEM_LIMIT(fine, ring);
    launch_pdl(fine, fine_grid, NWF * 32, ring, st, a, maps);
    LLSA_LAUNCH_OK("attn_fwd_fine_kernel");
    return loop_tc ? launch_attn_fwd_pooled_loop_tc(g, a, BH, st) : launch_attn_fwd_pooled_tc(g, a, BH, st);
  }
  const int n_smem = pooled_smem_tiles(a.p1_blocks + a.p2_blocks);
  const size_t smem = (size_t) n_smem * kBS * kSmemPitch * sizeof(bf16) * 2;
  LLSA_SMEM_LIMIT((attn_fwd_mma_kernel<NW>), smem);
  dim3 grid((unsigned) (a.nq1 / NW), (unsigned) (g->q->shape[0] * a.H));
  attn_fwd_mma_kernel<NW><<<grid, NW * 32, smem, st>>>(a, n_smem);
  LLSA_LAUNCH_OK("attn_fwd_mma_kernel");
  return LLSA_OK;
}

}  // namespace llsa
