"""Coarse selection over the list lengths where its kernels change, and the fused two-level selection against its two steps."""
import pytest
import torch

from helpers import topk_mismatch_rows
from llsa_b200 import ops, synth
from oracle import llsa_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# (BH, M, n): fewer keys than a 16-key block holds rows for, whole 64-key tiles (tensor cores: 16-row and, from 296 CTAs of 64 rows on,
# 64-row CTAs), ragged lists (scalar: below, at and past a 256-key chunk), rows that do not fill a tile
@pytest.mark.parametrize("BH,M,n", [(2, 64, 64), (3, 72, 128), (5, 4096, 320), (2, 40, 21), (3, 160, 160), (1, 300, 256 + 33), (2, 17, 1000)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("topk", [1, 8, 16])
def test_coarse_topk_shapes(BH, M, n, dtype, topk):
    gen = torch.Generator().manual_seed(1000 * n + M + topk)
    pq, pk = (torch.randn(1, BH, M, 64, generator=gen) * 0.25).to(dtype), (torch.randn(1, BH, n, 64, generator=gen) * 0.25).to(dtype)
    pk[:, :, n // 2] = pk[:, :, n // 3]                     # two equal columns: the smaller one first
    got = ops._coarse_topk(pq.to(DEV), pk.to(DEV), topk).cpu()
    want = O.gen_sparse_indices(pq, pk, topk)
    scores = (pq.float() @ pk.float().transpose(-1, -2)).to(dtype).float()
    # a bf16 score may round to the neighbouring value when its fp32 sum is taken in another order: one ulp of the largest scores (|s| < 4)
    differ, bad = topk_mismatch_rows(got, want, scores, margin=2.0 ** -6 if dtype == torch.bfloat16 else 1e-6)
    assert bad == 0 and differ <= max(2, 0.02 * BH * M)
    assert int(got.min()) >= 0 and int(got.max()) < n
    assert topk == 1 or (got.sort(-1).values.diff(dim=-1) > 0).all(), "duplicate block in a row"


# long lists and many rows: lists that end half way through a 128-key chunk (an odd and an even number of chunks), rows that do not fill a tile
@pytest.mark.parametrize("BH,M,n,topk", [(128, 40, 512, 8), (64, 130, 576, 8), (130, 40, 704, 5), (16, 1024, 1024, 4), (43, 300, 4160, 1), (129, 4, 8192, 8)])
def test_coarse_topk_of_long_lists(BH, M, n, topk):
    test_coarse_topk_shapes(BH, M, n, torch.bfloat16, topk)


@pytest.mark.parametrize("wait_limit", [0, 1])
@pytest.mark.parametrize("kind", ["ties", "equal", "nan", "-inf", "masked"])
@pytest.mark.parametrize("n", [512, 1088])
def test_coarse_topk_of_long_lists_orders_exact_scores(n, kind, wait_limit):
    _exact_scores(64, 200, n, kind, wait_limit)


def _exact_scores(BH, M, n, kind, wait_limit):
    """Small whole numbers: sums are exact in any order, so the order of a row is known, ties to the smaller column and NaN first.  A limit of one
    look makes the tcgen05 kernel's waits run out: its CTAs then select with scalar arithmetic."""
    from llsa_b200 import _lib
    gen = torch.Generator().manual_seed(n)
    pq, pk = torch.randint(-2, 3, (1, BH, M, 64), generator=gen).bfloat16(), torch.randint(-2, 3, (1, BH, n, 64), generator=gen).bfloat16()
    pq[..., 0] = 1
    if kind == "equal":
        pk[:] = pk[:, :, :1]
    elif kind == "nan":
        pk[:, :, ::97, 3] = float("nan")
        pq[:, :, 5, 7] = float("nan")
    elif kind == "-inf":
        pk[:, :, 40:n - 5, 0] = float("-inf")
    elif kind == "masked":
        pk[:, :, ::2] = 0
        pk[:, :, ::2, 0] = -3e38
    score = (pq.float() @ pk.float().transpose(-1, -2)).bfloat16().float()
    rank = torch.where(score.isnan(), torch.full_like(score, float("inf")), score)
    want = rank.sort(dim=-1, descending=True, stable=True).indices[..., :8].int()
    q, k, got = pq.to(DEV), pk.to(DEV), torch.full((1, BH, M, 8), -1, dtype=torch.int32, device=DEV)
    d = [_lib.desc(t) for t in (q, k, got)]
    _lib.check(_lib.lib().llsa_coarse_topk_bounded(*[_lib.ref(t) for t in d], 8, wait_limit, _lib.stream_ptr(torch.device(DEV))), "coarse_topk_bounded")
    assert torch.equal(got.cpu(), want)


# the tcgen05 kernel: its shortest list and the longest, lists that end half way through a 128-key chunk; few tiles, whose keys a cluster of eight, four or two
# CTAs shares (up to 32, 64 and 128), with shares of unlike length, and more than that
@pytest.mark.parametrize("BH,M,n,topk", [(1, 40, 2048, 8), (1, 300, 2112, 8), (2, 128, 4160, 5), (8, 500, 2048, 8), (9, 500, 2112, 8), (17, 512, 2176, 4),
                                         (129, 4, 2048, 8), (43, 300, 2112, 1), (1, 16, 65536, 8)])
def test_coarse_topk_on_tcgen05(BH, M, n, topk):
    test_coarse_topk_shapes(BH, M, n, torch.bfloat16, topk)


# tiles: a cluster of eight, four, two, none
@pytest.mark.parametrize("wait_limit", [0, 1])
@pytest.mark.parametrize("kind", ["ties", "equal", "nan", "-inf", "masked"])
@pytest.mark.parametrize("BH,n", [(2, 2048), (2, 2112), (40, 2112), (100, 2048), (129, 2112)])
def test_coarse_topk_on_tcgen05_orders_exact_scores(BH, n, kind, wait_limit):
    _exact_scores(BH, 8, n, kind, wait_limit)


# 512 tiles of 128 rows together; 32, 4 and 1 alone.  At these sizes a kernel that sums in another order chooses other blocks for one row or more.
@pytest.mark.parametrize("n,seed", [(512, 0), (1024, 1), (2048, 2), (4096, 3)])
def test_coarse_selection_of_a_row_depends_on_its_keys_alone(n, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    pq, pk = [(torch.randn(1, 16, m, 64, device=DEV, generator=gen) * 0.25).bfloat16() for m in (4096, n)]
    whole = ops._coarse_topk(pq, pk, 8)
    for h in range(16):
        assert torch.equal(whole[:, h:h + 1], ops._coarse_topk(pq[:, h:h + 1].contiguous(), pk[:, h:h + 1].contiguous(), 8)), h
    for r in (0, 16, 1024, 3984):
        for rows in (112, 512):
            part = pq[:, :2, r:r + rows].contiguous()
            assert torch.equal(whole[:, :2, r:r + rows], ops._coarse_topk(part, pk[:, :2].contiguous(), 8)), (r, rows)


def test_coarse_topk_zero_and_negative_scores_tie_and_order():
    """Scores of exactly zero of either sign tie, so the smaller column wins; all-negative rows come out in order."""
    pq, pk = torch.zeros(1, 1, 64, 64, dtype=torch.bfloat16), torch.zeros(1, 1, 128, 64, dtype=torch.bfloat16)
    pq[..., 0] = 1.0
    pk[0, 0, :, 0] = -torch.arange(128).float().to(torch.bfloat16) - 1
    pk[0, 0, 64:, 0] = -0.0
    got = ops._coarse_topk(pq.to(DEV), pk.to(DEV), 8).cpu()
    assert torch.equal(got, torch.arange(64, 72, dtype=torch.int32).expand(1, 1, 64, 8))
    pk[0, 0, 64:, 0] = -1000.0
    got = ops._coarse_topk(pq.to(DEV), pk.to(DEV), 8).cpu()
    assert torch.equal(got, torch.arange(8, dtype=torch.int32).expand(1, 1, 64, 8))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("N,topk,p_topk", [(2048, 8, 8), (5376, 8, 8), (16384, 8, 8), (16384, 16, 16), (24576, 4, 4), (40960, 16, 16), (73728, 8, 8)])
def test_select_two_level_is_its_two_steps(N, topk, p_topk, dtype):
    """One launch (level-2 lists of 8, 21, 64, 96, 160 keys) or two (288 keys): the bits of the coarse step followed by the refine step."""
    q, k = synth.gaussian_qkv(N + topk, 1, 2, N // 16, 64, n_tensors=2, dtype=dtype)
    pq, pk = q.to(DEV), k.to(DEV)
    pq2, pk2 = ops.mean_pool1d(pq, 16), ops.mean_pool1d(pk, 16)
    idx, pidx = ops._select_two_level(pq, pk, pq2, pk2, topk, p_topk, 16)
    assert torch.equal(pidx, ops._coarse_topk(pq2, pk2, p_topk))
    assert torch.equal(idx, ops._refine_topk(pq, pk, pidx, topk, p_topk, 16))
    want = O.compute_topk_indices_sparse(pq.cpu(), pk.cpu(), pidx.cpu().long(), topk, p_topk, 16)
    scores = pq.cpu().float() @ pk.cpu().float().transpose(-1, -2)
    differ, bad = topk_mismatch_rows(idx.cpu(), want, scores, margin=1e-5)       # fp32 sums of 64 products of size < 16 in another order
    assert bad == 0


@pytest.mark.parametrize("H,N", [(4, 47360), (5, 40960)])
def test_fp32_selection_of_one_wave_of_five_ctas_per_sm_and_of_more(H, N):
    """740 CTAs and 800: the lists of its two steps, and what every head has alone."""
    gen = torch.Generator(device=DEV).manual_seed(N)
    pq, pk = [torch.randn(1, H, N // 16, 64, device=DEV, generator=gen) for _ in range(2)]
    pq2, pk2 = ops.mean_pool1d(pq, 16), ops.mean_pool1d(pk, 16)
    idx, pidx = ops._select_two_level(pq, pk, pq2, pk2, 16, 16, 16)
    assert torch.equal(pidx, ops._coarse_topk(pq2, pk2, 16)) and torch.equal(idx, ops._refine_topk(pq, pk, pidx, 16, 16, 16))
    for h in range(H):
        alone = ops._select_two_level(*[t[:, h:h + 1].contiguous() for t in (pq, pk, pq2, pk2)], 16, 16, 16)
        assert torch.equal(alone[0], idx[:, h:h + 1]) and torch.equal(alone[1], pidx[:, h:h + 1])


# lists with repeats inside a row, every entry in one bucket, keys outside their range; one and several key ranges, 16 and 32 warps, T = 1
@pytest.mark.parametrize("BH,M,T,n,kind", [(1, 16, 8, 16, "uniform"), (3, 130, 6, 129, "uniform"), (2, 3000, 8, 3000, "one"), (1, 5000, 16, 5000, "hot"),
                                           (2, 300, 1, 1000, "uniform"), (60, 64, 8, 64, "hot"), (1, 16384, 8, 16384, "hot")])
def test_transpose_ranges(BH, M, T, n, kind):
    gen = torch.Generator().manual_seed(M + T)
    idx = torch.randint(0, n, (1, BH, M, T), generator=gen, dtype=torch.int32)
    if kind == "one":
        idx[:] = n - 1
    elif kind == "hot":
        idx[..., : T // 2] = torch.randint(0, 5, (1, BH, M, T // 2), generator=gen, dtype=torch.int32)
    off, flat = ops.transpose_indices(idx.to(DEV), n)
    e = torch.arange(M * T).expand(BH, -1)
    key, order = idx.reshape(BH, -1).long().sort(dim=1, stable=True)
    assert torch.equal(flat.cpu()[0].long(), e.gather(1, order) // T)
    assert torch.equal(off.cpu()[0, :, 1:].long(), torch.searchsorted(key, torch.arange(n).expand(BH, -1).contiguous(), right=True))
    assert int(off[..., 0].abs().max()) == 0
    # the pairs list, and what lies behind the last kept entry when keys are dropped
    bad = idx.clone()
    bad[:, :, M // 2] = n
    off, flat, (pairs, ranges), _ = ops._transpose(bad.to(DEV), n, torch.int32, True)
    kept = (M - 1) * T
    assert (off.cpu()[0, :, -1] == kept).all()
    assert torch.equal(pairs.cpu()[0, :, :kept] // T, flat.cpu()[0, :, :kept])
    assert (pairs.cpu()[0, :, :kept].sort(-1).values.diff(dim=-1) > 0).all()
    cut = ranges.cpu()[0, ..., 0]
    assert int(cut.min()) >= 0 and int(cut.max()) <= kept and (cut.diff(dim=-1) >= 0).all()


def test_index_transpose_of_many_heads():
    """More (batch, head) slices than the y axis of a launch grid holds."""
    heads, M, T, n = 70000, 2, 2, 8
    idx = torch.randint(0, n, (heads, 1, M, T), generator=torch.Generator().manual_seed(1), dtype=torch.int32)
    offsets, flat = [t.cpu() for t in ops.transpose_indices(idx.to(DEV), n)]
    counts = torch.nn.functional.one_hot(idx.long().view(heads, -1), n).sum(1)
    assert torch.equal(offsets[:, 0, 1:], counts.cumsum(-1)) and not offsets[..., 0].any()
    order = idx.view(heads, -1).sort(dim=-1, stable=True).indices          # entry positions by key, in their original order
    assert torch.equal(flat[:, 0], (order // T).int())


@pytest.mark.parametrize("n_kv", [64, 16384])
def test_index_transpose_without_the_pairs_list_and_scratch(n_kv):
    import ctypes as C

    from llsa_b200 import _lib
    B, H, M, T = 1, 2, 300, 8
    idx = torch.randint(0, n_kv, (B, H, M, T), generator=torch.Generator().manual_seed(n_kv), dtype=torch.int32).to(DEV)
    offsets, flat, (pairs, ranges), _ = ops._transpose(idx, n_kv, torch.int32, True)
    got = [torch.full_like(t, -7) for t in (offsets, flat, ranges)]
    d = [_lib.desc(t) for t in (idx, *got)]
    lib = _lib.lib()
    _lib.check(lib.llsa_transpose_indices_pairs(*[_lib.ref(t) for t in d[:3]], None, _lib.ref(d[3]), n_kv, None, 0, None, _lib.stream_ptr(torch.device(DEV))),
               "transpose_indices_pairs")
    assert all(torch.equal(a, b) for a, b in zip(got, (offsets, flat, ranges)))
    assert torch.equal(flat.long(), pairs.long() // T)
