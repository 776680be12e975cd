"""o and dq of lists whose fine and pooled keys are summed by two kernels: rounded to bf16 once, as where one kernel holds the sums in fp32."""
import pytest
import torch

import llsa_b200
from llsa_b200 import ops, synth

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _fp64(q, k, v, do, dbg):
    """o and dq of one (batch, head) in fp64, for the pooled tensors and lists of `dbg`."""
    n1, two = q.shape[0] // 16, "pk2" in dbg
    q, k, v, do = [t.double() for t in (q, k, v, do)]
    q.requires_grad_(True)
    level = {n: dbg[n][0, 0].double() for n in ("pk", "pv", "pk2", "pv2") if n in dbg}
    n2 = n1 // 16
    take = lambda t, blocks: t.view(-1, 16, 64)[blocks.long()].reshape(blocks.shape[0], -1, 64)
    out = []
    for b0 in range(0, n1, 128):
        rows = torch.arange(b0, min(b0 + 128, n1), device=q.device)
        fine = dbg["indices"][0, 0][rows]
        ks, vs, weights = [take(k, fine)], [take(v, fine)], [(fine.shape[1] * 16, 1.0)]
        if two:
            parents = dbg["p_indices"][0, 0][rows // 16]
            ks.append(take(level["pk"], parents)), vs.append(take(level["pv"], parents)), weights.append((parents.shape[1] * 16, 16.0))
        if two and n2 >= 64 or not two and n1 >= 64:
            every = ("pk2", "pv2", n2, 256.0) if two else ("pk", "pv", n1, 16.0)
            ks.append(level[every[0]].expand(len(rows), -1, -1)), vs.append(level[every[1]].expand(len(rows), -1, -1)), weights.append(every[2:])
        w = torch.cat([torch.full((n,), x, dtype=torch.float64, device=q.device) for n, x in weights]).log()
        s = q.view(n1, 16, 64)[rows] @ torch.cat(ks, 1).transpose(1, 2) / 8 + w
        o = (torch.softmax(s, -1) @ torch.cat(vs, 1)).reshape(-1, 64)
        o.backward(do[b0 * 16:b0 * 16 + len(o)])
        out.append(o.detach())
    return torch.cat(out), q.grad


# one level: 64 (dq alone: its forward has always been two kernels, as with 128 and 192 keys) and 160 pooled keys; two levels: 128
# gathered keys alone (dq), 128 + 96, 256 + 160 (one pass over the keys)
@pytest.mark.parametrize("N,topk,topk2,names", [(1024, 8, 0, ("dq",)), (2560, 8, 0, ("o", "dq")), (5376, 8, 8, ("dq",)), (24576, 8, 8, ("o", "dq")),
                                                (40960, 16, 16, ("o", "dq"))])
def test_rounded_once(N, topk, topk2, names, monkeypatch):
    q, k, v, do = [t.to(DEV) for t in synth.gaussian_qkv(N, 1, 1, N, 64, dtype=torch.bfloat16)]
    error = {}
    for one_kernel in (False, True):
        monkeypatch.setattr(ops, "_no_tcgen05", one_kernel)
        x = [t.detach().clone().requires_grad_(True) for t in (q, k, v)]
        dbg = llsa_b200.llsa_l2_debug(*x, topk, topk2, 16) if topk2 else llsa_b200.llsa_l1_debug(*x, topk, 16)
        dq, = torch.autograd.grad(dbg["o"], x[0], do)
        want = _fp64(q[0, 0], k[0, 0], v[0, 0], do[0, 0], dbg)
        error[one_kernel] = {n: float((g[0, 0].double() - w).norm() / w.norm()) for n, g, w in zip(("o", "dq"), (dbg["o"].detach(), dq), want)}
    # Both forms round P and dS to bf16 and the result once, but the one kernel's running maximum makes a few more of the large
    # probabilities exact: up to 1.7 % measured over lists of 96 to 1376 keys, N(0,1) and image-like inputs.  A result rounded twice has
    # variance 2^-18 / 12 times its weight more: 4 % to 14 % on these inputs.
    for name in names:
        assert error[False][name] <= 1.02 * error[True][name], (name, error)
