"""The key-loop tcgen05 kernels (forward, pooled dQ, pooled dK/dV) over pooled lists that end inside a chunk, against the oracle."""
import pytest
import torch

import llsa_b200
from llsa_b200 import ops, synth
from oracle import llsa_oracle as O
from test_gpu_parity import _oracle_l2_check, assert_bf16_close

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# gathered keys alone (fewer than 64 level-2 keys): a quarter, half, three quarters of a chunk, one, two, four chunks; level-2 tails of 32, 96 and
# 64 + 32 keys behind them
@pytest.mark.parametrize("B,H,N,topk,topk2", [(2, 3, 5376, 8, 8), (1, 2, 4096, 8, 2), (1, 2, 4096, 8, 4), (1, 1, 4096, 8, 6), (1, 2, 5120, 16, 16),
                                              (1, 1, 8192, 8, 32), (1, 2, 24576, 8, 8), (1, 1, 24576, 4, 4), (1, 1, 24576, 8, 2), (1, 1, 40960, 16, 16)])
def test_two_level_lists_vs_oracle(B, H, N, topk, topk2):
    q, k, v, do = synth.gaussian_qkv(N + topk2, B, H, N, 64, dtype=torch.bfloat16)
    _oracle_l2_check(llsa_b200, q, k, v, do, topk1=topk, topk2=topk2, label="N=%d top-%d/%d" % (N, topk, topk2))


@pytest.mark.parametrize("one_pass", [True, False])
@pytest.mark.parametrize("B,H,N", [(2, 3, 1536), (1, 2, 2560), (1, 2, 5632), (3, 1, 8704)])      # 96, 160, 352, 544 pooled keys
def test_one_level_lists_vs_oracle(B, H, N, one_pass, monkeypatch):
    monkeypatch.setattr(ops, "_one_pass_pooled", one_pass)
    q, k, v, do = synth.gaussian_qkv(N, B, H, N, 64, dtype=torch.bfloat16)
    qg, kg, vg = [t.to(DEV).requires_grad_(True) for t in (q, k, v)]
    dbg = llsa_b200.llsa_l1_debug(qg, kg, vg, 8, 16)
    idx, pk, pv = dbg["indices"].cpu(), dbg["pk"].cpu(), dbg["pv"].cpu()
    o_ref, lse_ref = O.attn_fwd_l1(q, k, v, pk, pv, idx, faithful=False)
    assert_bf16_close(dbg["o"].detach(), o_ref, "o")
    assert float((dbg["lse"].cpu() - lse_ref).abs().max()) < 2e-2
    dbg["o"].backward(do.to(DEV))
    dq, dk, dv, dpk, dpv = O.attn_bwd_l1(do, q, k, v, pk, pv, o_ref.float(), lse_ref, idx, faithful=False)
    assert_bf16_close(qg.grad, dq, "dq")
    assert_bf16_close(kg.grad, dk + O.mean_pool1d_bwd(dpk, 16), "dk")
    assert_bf16_close(vg.grad, dv + O.mean_pool1d_bwd(dpv, 16), "dv")


# the two sides of the line up to which the dQ epilogue requests its remainder ahead: 288 and 320 keys are five jobs, 352 and two levels' 256 + 96 six
LINE = [(4608, 8, 0), (5120, 8, 0), (5632, 8, 0), (24576, 8, 16)]


@pytest.mark.parametrize("N,topk,topk2", LINE)
def test_remainder_of_dq_at_the_line(N, topk, topk2, monkeypatch):
    """The one-kernel form's error is the measure, as for the other lists: a remainder left out or in the wrong place is beyond it."""
    from test_rounding import test_rounded_once as check
    check(N, topk, topk2, ("dq",), monkeypatch)


@pytest.mark.parametrize("N,topk,topk2", LINE[1:])
def test_dq_of_a_head_does_not_depend_on_its_tiles_neighbours(N, topk, topk2):
    """Three and more tiles per CTA against the same head alone (one tile, or two): what is requested ahead belongs to the next tile."""
    H = max(2, 148 * 128 * 3 // N + 1)
    x = [t.to(DEV) for t in synth.gaussian_qkv(N + topk2, 1, H, N, 64, dtype=torch.bfloat16)]

    def dq(h0, h1):
        q, k, v, do = [t[:, h0:h1].detach().clone() for t in x]
        q.requires_grad_(True)
        o = llsa_b200.llsa_l2(q, k, v, topk, topk2, 16) if topk2 else llsa_b200.llsa_l1(q, k, v, topk, 16)
        return torch.autograd.grad(o, q, do)[0]

    every = dq(0, H)
    for h in (0, H - 1):
        assert torch.equal(every[:, h:h + 1], dq(h, h + 1)), h


# the lines between two and three softmax groups of the forward: 256 and 384 keys without a remainder, 448 and 480 with one
@pytest.mark.parametrize("one_pass", [True, False])
@pytest.mark.parametrize("N", [4096, 6144, 7168, 7680])
def test_forward_on_both_sides_of_the_group_line(N, one_pass, monkeypatch):
    """Against the oracle, and with three and more tiles per CTA what the first and last head give alone.  Which group takes a tile's first job
    depends on the tile's place, and with it the order of the fp32 sum of a row's three or two partial sums: 2^-23 of it, which moves one o in
    2^-23 / 2^-8 = 2^-15 over a rounding boundary of bf16, by 2^-8 at most: 2^-15.5 in the 2-norm.  A row or a tile mixed up is of order one."""
    test_one_level_lists_vs_oracle(1, 1, N, one_pass, monkeypatch)
    H = 148 * 128 * 3 // N + 1
    q, k, v, _ = [t.to(DEV) for t in synth.gaussian_qkv(N + 1, 1, H, N, 64, dtype=torch.bfloat16)]
    with torch.no_grad():
        every = llsa_b200.llsa_l1(q, k, v, 8, 16)
        for h in (0, H - 1):
            alone = llsa_b200.llsa_l1(*[t[:, h:h + 1].contiguous() for t in (q, k, v)], 8, 16).float()
            assert float((every[:, h:h + 1].float() - alone).norm() / alone.norm()) < 2 ** -13, h


def test_tail_keys_of_the_next_head_do_not_leak():
    """A chunk's rows behind the end of a head's list belong to the next head: NaN and infinities there must stay there."""
    q, k, v, do = [t.to(DEV) for t in synth.gaussian_qkv(5, 1, 2, 2560, 64, dtype=torch.bfloat16)]
    want = [t.detach().clone().requires_grad_(True) for t in (q[:, :1], k[:, :1], v[:, :1])]
    o_want = llsa_b200.llsa_l1(*want, 8, 16)
    o_want.backward(do[:, :1])
    k2, v2 = k.clone(), v.clone()
    k2[:, 1], v2[:, 1] = float("inf"), float("nan")
    got = [t.detach().clone().requires_grad_(True) for t in (q, k2, v2)]
    o = llsa_b200.llsa_l1(*got, 8, 16)
    o.backward(do)
    assert torch.equal(o[:, :1], o_want) and torch.equal(got[0].grad[:, :1], want[0].grad)
    for i in (1, 2):      # fp32 reductions: the order of the sums may differ
        assert float((got[i].grad[:, :1].float() - want[i].grad.float()).norm() / want[i].grad.float().norm()) < 1e-3


def test_marks_are_those_of_the_last_debug_call():
    """A production call leaves no marks (nor their memory) behind, and a debug call whose list needs none says so."""
    q, k, v, _ = [t.to(DEV) for t in synth.gaussian_qkv(7, 1, 2, 16384, 64, dtype=torch.bfloat16)]
    llsa_b200.llsa_l1_debug(q, k, v, 8, 16)                                  # 1024 pooled keys: one pass, marks
    marks = ops._last_fwd_redo
    assert marks.numel() * 4 == 2 * 16384 and not marks.any()
    short = [t[:, :, :5632].contiguous() for t in (q, k, v)]
    llsa_b200.llsa_l1(*short, 8, 16)
    assert ops._last_fwd_redo.data_ptr() == marks.data_ptr()
    llsa_b200.llsa_l1_debug(*short, 8, 16)
    assert ops._last_fwd_redo.numel() * 4 == 2 * 5632
    llsa_b200.llsa_l2_debug(q, k, v, 8, 8, 16)                               # 192 pooled keys: all at once
    assert ops._last_fwd_redo is None
