"""The layer with the q / k preparation in front, as a caller makes it: table types, absent norms and tables, frozen weights."""
import pytest
import torch

import llsa_b200
from llsa_b200 import ops, synth

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
EPS = 1e-5


def _inputs(N, seed=3):
    q, k, v, do = [t.to(DEV) for t in synth.gaussian_qkv(seed, 1, 2, N, 64, dtype=torch.bfloat16)]
    gen = torch.Generator().manual_seed(seed)
    ang = torch.rand(N, 32, generator=gen) * 6.3
    table = torch.stack([ang.sin(), ang.cos()], -1).reshape(N, 64).to(DEV)
    wq, wk = (1 + 0.2 * torch.randn(2, 64, generator=gen)).to(DEV)
    return q, k, v, do, table, wq, wk


def _norm_backward(x, w, g):
    x, g = x.double(), g.double()
    rstd = torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS)
    xh, gw = x * rstd, g * w.double()
    return rstd * (gw - xh * (gw * xh).mean(-1, keepdim=True)), (g * xh).sum((0, 1, 2))


@pytest.mark.parametrize("table_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,two_level", [(2048, False), (4096, True)])
def test_norm_and_rotation_backward_with_the_table_as_given(N, two_level, table_dtype):
    """dq and the norm's weight gradient against the stand-alone rotation with the same table (bf16 data, fp32 table: products rounded to
    fp32, not with a table cut to bf16) and the norm's gradient in fp64."""
    q, k, v, do, table, wq, wk = _inputs(N)
    table = table.to(table_dtype)
    x, w = [t.detach().clone().requires_grad_(True) for t in (q, k, v)], [t.clone().requires_grad_(True) for t in (wq, wk)]
    layer = llsa_b200.llsa_l2_rms_rope if two_level else llsa_b200.llsa_l1_rms_rope
    layer(*x, *w, table, EPS).backward(do)
    # the operator on q and k prepared beforehand
    prepared = [llsa_b200.my_rope_fn(ops.rms_norm(t, s, EPS), table.to(q.dtype)).detach().requires_grad_(True) for t, s in ((q, wq), (k, wk))]
    plain = llsa_b200.llsa_l2 if two_level else llsa_b200.llsa_l1
    dqr, = torch.autograd.grad(plain(*prepared, v), prepared[:1], do)
    dq, dw = _norm_backward(q, wq, ops._rope_bwd_op(dqr, table))
    assert ((x[0].grad.double() - dq).abs() <= 2.0 ** -8 * dq.abs() + 2e-5 * float(dq.abs().max())).all()       # one rounding to bf16
    assert float((w[0].grad.double() - dw).norm() / dw.norm()) < 1e-5                                           # fp32 sums


# which of wq, wk and the table are given; which of the inputs take a gradient; which gradients are asked for
@pytest.mark.parametrize("given,train,ask", [
    ("wq wk table", "q k v wq wk", "q k wq wk"), ("wq wk", "q k v wq wk", "q wq wk"), ("wq wk", "q k v", "q k"), ("wq wk", "q k v wq", "q wq"),
    ("wq wk", "q k v wk", "k wk"), ("wq wk", "wk", "wk"), ("wq table", "q k v wq", "q wq"), ("wk table", "q k v wk", "q k wk"), ("wk table", "q k v", "q"),
    ("wq", "wq", "wq"), ("wk", "q k v wk", "q wk"), ("wq wk table", "q k v wk", "q wk"), ("wq wk table", "q k v wq wk", "q")])
def test_absent_norms_and_tables_frozen_weights(given, train, ask):
    """Gradients of every form of the call against the operator on q and k prepared beforehand."""
    given, train, ask = given.split(), train.split(), ask.split()
    q, k, v, do, table, wq, wk = _inputs(4096)
    table = table.to(q.dtype)
    t = dict(q=q, k=k, v=v, wq=wq if "wq" in given else None, wk=wk if "wk" in given else None)
    x = {n: s.detach().clone().requires_grad_(n in train) if s is not None else None for n, s in t.items()}
    o = llsa_b200.llsa_l2_rms_rope(x["q"], x["k"], x["v"], x["wq"], x["wk"], table if "table" in given else None, EPS)
    got = dict(zip(ask, torch.autograd.grad(o, [x[n] for n in ask], do)))
    prepared = {}
    for n, w in (("q", t["wq"]), ("k", t["wk"])):
        y = ops.rms_norm(t[n], w, EPS) if w is not None else t[n]
        prepared[n] = (llsa_b200.my_rope_fn(y, table) if "table" in given else y).detach().clone().requires_grad_(True)
    want_o = llsa_b200.llsa_l2(prepared["q"], prepared["k"], v)
    assert torch.equal(o, want_o)
    grads = dict(zip("qk", torch.autograd.grad(want_o, [prepared["q"], prepared["k"]], do)))
    for n, w in (("q", t["wq"]), ("k", t["wk"])):
        g = ops._rope_bwd_op(grads[n], table) if "table" in given else grads[n]
        dx, dw = _norm_backward(t[n], w, g) if w is not None else (g.double(), None)
        # one rounding to bf16 (2^-9 of a value at most) on top of the sums of the pooled-key gradients, whose order differs from call to call
        if n in got:
            assert float((got[n].double() - dx).norm() / dx.norm()) < 2.0 ** -8
        if "w" + n in got:
            assert float((got["w" + n].double() - dw).norm() / dw.norm()) < 1e-4


@pytest.mark.parametrize("which", ["q", "v", "wk"])
def test_forward_mode_is_refused(which):
    import torch.autograd.forward_ad as fw
    q, k, v, do, table, wq, wk = _inputs(2048)
    x = dict(q=q, k=k, v=v, wq=wq, wk=wk)
    with fw.dual_level():
        x[which] = fw.make_dual(x[which], torch.ones_like(x[which]))
        with pytest.raises(NotImplementedError):
            llsa_b200.llsa_l1_rms_rope(*x.values(), table.to(q.dtype), EPS)


# 4,032, 4,096, 24,576 and 25,600 query blocks: on both sides of the lines between which the values are pooled beside the selection
@pytest.mark.parametrize("B,H,N", [(2, 6, 5376), (1, 8, 8192), (3, 8, 16384), (5, 5, 16384)])
def test_values_pooled_beside_the_selection(B, H, N):
    """Pooled values and output of the layer are those of its parts called one by one, bit for bit, on new values at every call and in a graph."""
    gen = torch.Generator(device=DEV).manual_seed(N + B)
    q, k, v = [torch.randn(B, H, N, 64, device=DEV, generator=gen).bfloat16() for _ in range(3)]

    def parts():
        (pq, pk, pv), (pq2, pk2, pv2) = ops.pool_pyramid([q, k, v], 16, 2)
        idx, pidx = ops._select_two_level(pq, pk, pq2, pk2, 8, 8, 16)
        return idx, pv, pv2, ops._attn_fwd(q, k, v, pk, pv, pk2, pv2, idx, pidx, 8, 8, 16, 16.0, 256.0)[0]

    for _ in range(3):
        got, (idx, pv, pv2, o) = llsa_b200.llsa_l2_debug(q, k, v), parts()
        assert torch.equal(got["o"], o)      # an attention stage that ran ahead of the values' pooling would have read the last call's
        assert torch.equal(got["indices"], idx.to(got["indices"].dtype)) and torch.equal(got["pv"], pv) and torch.equal(got["pv2"], pv2)
        v.normal_(generator=gen)
    want = llsa_b200.llsa_l2(q, k, v)
    x = [t.detach().clone() for t in (q, k, v)]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side), torch.no_grad():
        llsa_b200.llsa_l2(*x)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            o = llsa_b200.llsa_l2(*x)
    for t in x:
        t.zero_()
    graph.replay()
    for t, s in zip(x, (q, k, v)):
        t.copy_(s)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(o, want)
