"""Fine dK/dV kernel against the oracle: windows drawn by the warps of a CTA (lists of 4,736 ranges and more), equal spans of the entries (shorter
ones)."""
import ctypes as C

import pytest
import torch

import llsa_b200
from llsa_b200 import synth
from oracle import llsa_oracle as O
from test_gpu_parity import rel_l2

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _close(got, ref, name):
    """bf16 operands (Q, K, V, P, dS) and a bf16 result: every rounding is relative, 2^-9 of the value or of a term of its sum, so the error
    scales with the largest value of the tensor.  The sums have random signs: 5 x 2^-9 = 1e-2 covers five such roundings in the norm and
    2e-2 of the largest value ten in one element."""
    got, ref = got.detach().float().cpu(), ref.detach().float().cpu()
    assert rel_l2(got, ref) <= 1e-2, name
    assert float((got - ref).abs().max()) <= 2e-2 * max(1.0, float(ref.abs().max())), name


# 32 and 3 ranges per head (an odd number leaves a window of one range); hot: key blocks every query block selects, i.e. lists of N / 16
# entries that are cut between windows and inside them, next to blocks nobody selects
@pytest.mark.parametrize("B,H,N,topk,hot", [(37, 4, 2048, 8, ()), (37, 4, 2048, 8, (3,)), (37, 4, 2048, 8, (0, 1, 127)), (264, 6, 768, 2, ()),
                                            (264, 6, 768, 2, (3,)), (264, 6, 768, 2, (0, 47))])
def test_persistent_form_vs_oracle(B, H, N, topk, hot):
    q, k, v, do = synth.gaussian_qkv(N + len(hot), 2, H, N, 64, dtype=torch.bfloat16)
    u = torch.ones(64) * 0.35
    if hot:
        q = (q.float() + u).to(torch.bfloat16)
        for j in hot:
            k[:, :, 16 * j:16 * j + 16] = (k[:, :, 16 * j:16 * j + 16].float() + 4 * u).to(torch.bfloat16)
    rep = (B + 1) // 2
    Q, K, V, DO = [t.to(DEV).repeat(rep, 1, 1, 1)[:B].contiguous() for t in (q, k, v, do)]
    Q, K, V = [t.requires_grad_(True) for t in (Q, K, V)]
    dbg = llsa_b200.llsa_l1_debug(Q, K, V, topk, 16)
    dbg["o"].backward(DO)
    idx, pk, pv = [dbg[n][:2].cpu() for n in ("indices", "pk", "pv")]
    assert all(bool((idx == j).any(-1).all()) for j in hot)
    o_ref, lse_ref = O.attn_fwd_l1(q, k, v, pk, pv, idx, faithful=False)
    dq, dk, dv, dpk, dpv = O.attn_bwd_l1(do, q, k, v, pk, pv, o_ref.float(), lse_ref, idx, faithful=False)
    last = slice(2 * (rep - 1), B)                        # the same inputs again at the end of the batch
    for sl, n in ((slice(0, 2), 2), (last, B - 2 * (rep - 1))):
        _close(Q.grad[sl], dq[:n], "dq")
        _close(K.grad[sl], (dk + O.mean_pool1d_bwd(dpk, 16))[:n], "dk")
        _close(V.grad[sl], (dv + O.mean_pool1d_bwd(dpv, 16))[:n], "dv")


# spans: of 64 entries (a problem of fewer than 256), the shortest spans on some of the SMs, spans of two lengths on all of them, which begin and end
# inside buckets and inside heads; hot: a bucket that reaches over many spans, of one head and of every head
@pytest.mark.parametrize("B,H,N,topk,hot", [(2, 1, 256, 2, ()), (2, 1, 256, 8, ()), (3, 2, 768, 6, ()), (3, 2, 768, 6, (3,)), (2, 2, 1024, 8, (0, 63)),
                                            (9, 7, 2048, 8, ()), (9, 7, 2048, 8, (0, 1, 127)), (21, 11, 1024, 8, (5,))])
def test_spans_vs_oracle(B, H, N, topk, hot):
    test_persistent_form_vs_oracle(B, H, N, topk, hot)


@pytest.mark.parametrize("B,H,N", [(1, 2, 1024), (4, 6, 4096)])
def test_scratch_of_one_window_per_64_entries_is_enough(B, H, N):
    """llsa_attn_bwd with the least dkv_partial it accepts, through the C interface: fewer and longer spans, the same gradients."""
    from llsa_b200 import _lib
    L, dev = _lib.lib(), torch.device(DEV)
    gen = torch.Generator(device=DEV).manual_seed(N)
    q, k, v, do = [torch.randn(B, H, N, 64, device=DEV, generator=gen).bfloat16() for _ in range(4)]
    dbg = llsa_b200.llsa_l1_debug(q, k, v, 8, 16)
    idx, n1, E, S = dbg["indices"].int().contiguous(), N // 16, N // 16 * 8, L.llsa_transpose_range_entries(B, H, N // 16, 8)
    assert S == 16
    i32, f32 = dict(dtype=torch.int32, device=DEV), dict(device=DEV)
    t = dict(q=q, k=k, v=v, pk=dbg["pk"], pv=dbg["pv"], indices=idx, o=dbg["o"], lse=dbg["lse"], d_o=do, delta=torch.empty(B, H, N, **f32),
             offsets=torch.empty(B, H, n1 + 1, **i32), flat=torch.empty(B, H, E, **i32), flat_ranges=torch.empty(B, H, -(-E // S), 2, **i32),
             dpk_acc=torch.empty(B, H, n1, 64, **f32), dpv_acc=torch.empty(B, H, n1, 64, **f32), remainder=torch.empty_like(q))
    d = {n: _lib.desc(x) for n, x in t.items()}
    _lib.check(L.llsa_transpose_indices_pairs(*[_lib.ref(d[n]) for n in ("indices", "offsets", "flat")], None, _lib.ref(d["flat_ranges"]), n1, None, 0, None,
                                              _lib.stream_ptr(dev)), "transpose")
    least, full, got = B * H * -(-E // 64) * 4096, L.llsa_attn_bwd_partial_elems(B, H, N, 8), {}
    assert least < full
    for n in (least, full, least - 4096):
        out = [torch.full_like(q, float("nan")) for _ in range(3)]
        partial = torch.empty(1, 1, n // 4096, 4096, **f32)
        od, pd = [_lib.desc(x) for x in out], _lib.desc(partial)
        a = _lib.LlsaAttnArgs()
        for name, x in list(d.items()) + list(zip(("dq", "dk", "dv"), od)) + [("dkv_partial", pd)]:
            setattr(a, name, _lib.ptr(x))
        a.topk, a.block_size, a.token_weight, a.kv_weight, a.fold_pool_bwd = 8, 16, 16.0, 16.0, 1
        rc = L.llsa_attn_bwd(C.byref(a), _lib.stream_ptr(dev))
        torch.cuda.synchronize()
        assert (rc == 0) == (n >= least), (n, rc)
        got[n] = [x.float() for x in out]
    for x, y in zip(got[least], got[full]):      # fp32 sums meet in another order, then one rounding to bf16
        assert float((x - y).norm() / y.norm()) < 2e-3
