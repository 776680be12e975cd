"""Views whose rows lie on top of one another: keys shared by heads or batches, a gradient shared by tokens."""
import pytest
import torch

import llsa_b200
from llsa_b200 import synth

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# single-shot pooled kernels, key-loop kernels, scalar kernels
@pytest.mark.parametrize("N,two_level,dtype", [(16384, True, torch.bfloat16), (5632, False, torch.bfloat16), (1024, False, torch.float32)])
@pytest.mark.parametrize("dim", [0, 1])
def test_expanded_equals_contiguous(N, two_level, dtype, dim):
    B, H = 2, 3
    q, k, v, do = [t.to(DEV) for t in synth.gaussian_qkv(N + dim, B, H, N, 64, dtype=dtype)]
    k, v = [t.narrow(dim, 0, 1).expand(B, H, N, 64) for t in (k, v)]
    do = do[:, :, :1].expand(B, H, N, 64)                                   # what o.mean(2) sends back, up to its factor
    call = llsa_b200.llsa_l2 if two_level else llsa_b200.llsa_l1
    out = []
    for copy in (False, True):
        x = [(t.contiguous() if copy else t).detach().requires_grad_(True) for t in (q, k, v)]
        o = call(*x)
        out.append((o,) + torch.autograd.grad(o, x, do.contiguous() if copy else do))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    for a, b in zip(out[0][2:], out[1][2:]):                                # sums of the pooled-key gradients: their order differs from call to call
        assert float((a.float() - b.float()).norm() / b.float().norm()) < (1e-5 if dtype == torch.float32 else 1e-3)


def test_overlapping_tokens():
    """Every token's row begins a quarter row behind the one before it."""
    N = 4096
    flat = torch.randn(2, 16 * N + 64, generator=torch.Generator().manual_seed(2)).to(DEV, torch.bfloat16)
    k = flat.as_strided((1, 2, N, 64), (0, 16 * N + 64, 16, 1))
    q, v = [torch.randn(1, 2, N, 64, device=DEV, dtype=torch.bfloat16) for _ in range(2)]
    assert torch.equal(llsa_b200.llsa_l1(q, k, v), llsa_b200.llsa_l1(q, k.contiguous(), v))
