"""What a forward leaves behind whose bounded mbarrier waits run out (forced here by a poll limit of a few looks): with device checks off, a NaN in
lse is the only sign of it, so every row must hold its final value or NaN.  The fine part's own lse, which the pooled stage finds there, and what
an earlier call left in that memory look plausible and are neither."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _lse(levels, q, k, v):
    import llsa_b200 as L
    with torch.no_grad():
        return (L.llsa_l1_debug(q, k, v, 8, 16) if levels == 1 else L.llsa_l2_debug(q, k, v, 8, 8, 16))["lse"]


def _inputs(levels, B, H, N):
    gen = torch.Generator(device=DEV).manual_seed(N + levels)
    return [torch.randn((B, H, N, 64), generator=gen, device=DEV).bfloat16() for _ in range(3)]


def _check(levels, x, limit, monkeypatch):
    """-> rows left as NaN by a call under the poll limit; every other row is final, and so is the call after it."""
    from llsa_b200 import ops
    want = _lse(levels, *x).clone()
    _lse(levels, -x[0], x[1], x[2])          # so that what the limited call finds in memory is another call's
    monkeypatch.setattr(ops, "_wait_limit", limit)
    lse = _lse(levels, *x)
    torch.cuda.synchronize()
    monkeypatch.setattr(ops, "_wait_limit", 0)
    assert bool((lse.isnan() | (lse == want)).all()), int((~lse.isnan() & (lse != want)).sum())
    assert torch.equal(_lse(levels, *x), want)
    return int(lse.isnan().sum())


# key-loop pooled forward, one and two levels, one pass and two, two and three softmax groups, three to seven tiles per CTA; the single-shot one, ten
@pytest.mark.parametrize("levels,B,H,N,one_pass", [(1, 2, 8, 4096, True), (1, 2, 4, 16384, True), (1, 2, 4, 16384, False), (2, 1, 2, 65536, True), (2, 2, 6, 16384, True)])
def test_every_row_behind_an_expired_wait_of_the_pooled_forward_is_nan(levels, B, H, N, one_pass, monkeypatch):
    """A limit that the fine forward's waits keep and the pooled one's do not: the tiles behind a CTA's first unfinished one included."""
    from llsa_b200 import ops
    monkeypatch.setattr(ops, "_one_pass_pooled", one_pass)
    assert _check(levels, _inputs(levels, B, H, N), 8, monkeypatch) > 0


@pytest.mark.parametrize("limit", [8, 16, 20, 24, 28, 32, 36, 48])
def test_rows_marked_for_a_round_that_an_expired_wait_cuts_short_are_nan(limit, monkeypatch):
    """Logits in the hundreds: many rows are left to the second round, which never comes, or not to its end."""
    from llsa_b200 import ops, synth
    q, k, v = synth.correlated_qkv(51, 1, 2, 65536, 64, dtype=torch.bfloat16, n_tensors=3)
    x = [(q.float() * 12).to(DEV, torch.bfloat16), (k.float() * 12).to(DEV, torch.bfloat16), v.to(DEV)]
    _check(2, x, limit, monkeypatch)
    assert int(ops._last_fwd_redo.view(torch.uint8)[:2 * 65536].sum()) > 0


@pytest.mark.parametrize("levels,B,H,N", [(1, 2, 4, 16384), (2, 1, 2, 65536), (2, 2, 6, 16384)])
def test_every_row_behind_an_expired_wait_of_the_fine_forward_is_nan(levels, B, H, N, monkeypatch):
    """A limit of one: most of the fine forward's copies have not landed at the first look, and nothing writes those rows."""
    assert _check(levels, _inputs(levels, B, H, N), 1, monkeypatch) > 0


# key-loop dQ and dense dK/dV at one level, with the gathered dK/dV at two, lists that come with a remainder; the single-shot backward.  A limit of
# four: the fine stages' waits mostly keep it, those of a tile of many jobs do not
@pytest.mark.parametrize("levels,B,H,N,limits", [(1, 2, 6, 1024, (1,)), (1, 1, 4, 16384, (1, 4)), (2, 1, 3, 40960, (1, 4)), (2, 1, 2, 65536, (1, 4)),
                                                 (2, 1, 6, 16384, (1,))])
def test_expired_waits_of_the_backward_are_reported(levels, B, H, N, limits, monkeypatch):
    """The kernels leave their loops, give their tensor memory back and report it; the next backward is right again."""
    import llsa_b200 as L
    from llsa_b200 import ops
    q, k, v = _inputs(levels, B, H, N)
    do = torch.ones_like(q)
    q.requires_grad_(True)

    def forward():
        return L.llsa_l1(q, k, v, 8, 16) if levels == 1 else L.llsa_l2(q, k, v, 8, 8, 16)

    want, = torch.autograd.grad(forward(), q, do)
    for limit in limits:
        o = forward()
        torch.cuda.synchronize()
        monkeypatch.setattr(ops, "_wait_limit", limit)
        L.set_device_checks(True)
        ops._native()                # hands the settings over: the backward runs without a call of this module's
        try:
            with pytest.raises(RuntimeError, match="bounded wait"):
                torch.autograd.grad(o, q, do)
        finally:
            monkeypatch.setattr(ops, "_wait_limit", 0)
            L.set_device_checks(False)
            ops._native()
        torch.cuda.synchronize()
        again, = torch.autograd.grad(forward(), q, do)
        assert torch.equal(again, want)
