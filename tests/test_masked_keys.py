"""Keys masked by very low values: scores of -inf in whole blocks, in the whole share of a warp, in every pooled key of a row."""
import pytest
import torch

import llsa_b200
from llsa_b200 import ops
from oracle import llsa_oracle as O
from helpers import rel_l2

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _check(q, k, v, do, two_level, tol):
    x = [t.to(DEV).requires_grad_(True) for t in (q, k, v)]
    dbg = llsa_b200.llsa_l2_debug(*x, 8, 8, 16) if two_level else llsa_b200.llsa_l1_debug(*x, 8, 16)
    dbg["o"].backward(do.to(DEV))
    low = {n: t.detach().cpu() for n, t in dbg.items()}
    if two_level:
        args = (low["pk"], low["pv"], low["pk2"], low["pv2"])
        o, lse = O.attn_fwd_l2(q, k, v, *args, low["indices"], low["p_indices"].long(), faithful=False)
        dv = O.attn_bwd_l2(do, q, k, v, *args, o.float(), lse, low["indices"], low["p_indices"].long(), faithful=False)
        dv = dv[2] + O.mean_pool1d_bwd(dv[4] + O.mean_pool1d_bwd(dv[6], 16), 16)
    else:
        o, lse = O.attn_fwd_l1(q, k, v, low["pk"], low["pv"], low["indices"], faithful=False)
        dv = O.attn_bwd_l1(do, q, k, v, low["pk"], low["pv"], o.float(), lse, low["indices"], faithful=False)
        dv = dv[2] + O.mean_pool1d_bwd(dv[4], 16)
    assert torch.isfinite(o.float()).all() and torch.isfinite(dv).all()
    assert rel_l2(low["o"], o) < tol and rel_l2(low["lse"], lse) < tol and rel_l2(x[2].grad, dv) < tol
    for t in x:
        assert torch.isfinite(t.grad.float()).all()


def _inputs(N, dtype, masked, value):
    gen = torch.Generator().manual_seed(N)
    q, k = [torch.rand(1, 2, N, 64, generator=gen) + 0.5 for _ in range(2)]
    v, do = [torch.randn(1, 2, N, 64, generator=gen) for _ in range(2)]
    k[:, :, masked] = value
    return [t.to(dtype) for t in (q, k, v, do)]


# fp32 sums in another order, 1e-5; bf16 operands of the products, 1e-2 (the bounds of the parity tests)
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 1e-2)])
@pytest.mark.parametrize("N,two_level", [(1024, False), (2560, False), (4096, True)])
def test_all_but_four_blocks_masked(N, two_level, dtype, tol):
    """Half of the selected blocks and most pooled blocks hold nothing but scores of -inf."""
    q, k, v, do = _inputs(N, dtype, slice(64, None), -1e37)
    _check(q, k, v, do, two_level, tol)


@pytest.mark.parametrize("one_pass", [True, False])
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 1e-2)])
@pytest.mark.parametrize("N", [2560, 5632])
def test_one_token_of_every_block_masked(N, dtype, tol, one_pass, monkeypatch):
    """Every pooled key scores -inf, every selected block has fifteen keys that do not."""
    monkeypatch.setattr(ops, "_one_pass_pooled", one_pass)
    q, k, v, do = _inputs(N, dtype, slice(3, None, 16), -3e38)
    _check(q, k, v, do, False, tol)
