"""The layer operators under torch.compile and the checks of torch.library: traced whole, shape functions as the kernels allocate."""
import subprocess
import sys

import pytest
import torch

import llsa_b200
from llsa_b200 import ops, synth

DEV = "cuda:0"

# a fresh process: the first call of the library is the traced one
_FIRST_CALL = """
import torch, llsa_b200
from llsa_b200 import synth
q, k, v, do = [t.cuda() for t in synth.gaussian_qkv(1, 1, 2, 4096, 64, dtype=torch.bfloat16)]
table = torch.ones(4096, 64, device="cuda", dtype=torch.bfloat16)
w = torch.ones(64, device="cuda", requires_grad=True)
for call in (lambda *x: llsa_b200.llsa_l2(*x), lambda *x: llsa_b200.llsa_l1_rope(*x, table), lambda *x: llsa_b200.llsa_l2_rms_rope(*x, w, w, table)):
    x = [t.clone().requires_grad_(True) for t in (q, k, v)]
    o = torch.compile(lambda *x: call(*x) * 2, fullgraph=True, backend="aot_eager")(*x)
    want = call(*x) * 2
    assert torch.equal(o, want)
    got, want = [torch.autograd.grad(t, x, do) for t in (o, want)]
    # dq and dv repeat exactly or up to the order of fp32 sums in front of a rounding to bf16
    assert all(float((a.float() - b.float()).norm() / b.float().norm()) < 1e-3 for a, b in zip(got, want))
"""


@pytest.mark.gpu
def test_whole_graph_compile_of_a_first_call():
    r = subprocess.run([sys.executable, "-c", _FIRST_CALL], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]


def _operands(layout, N=2048, dtype=torch.bfloat16):
    q, k, v, do = [t.to(DEV) for t in synth.gaussian_qkv(1, 1, 2, N, 64, dtype=dtype)]
    if layout == "bnhd":
        q, k, v, do = [t.transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k, v, do)]
    if layout == "expanded":
        k, v = [t[:, :1].expand(1, 2, N, 64) for t in (k, v)]
    if layout == "offset":                            # rows that no kernel takes as they are
        q = torch.cat([q, q], -1)[..., 8:72]
    return [t.detach().requires_grad_(True) for t in (q, k, v)] + [do]


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["bhnd", "bnhd", "expanded", "offset"])
def test_operators_as_torch_library_checks_them(layout):
    """Shape functions, schemas (no output shares memory with another or with an input) and autograd registration."""
    ops._ready()
    L = torch.ops.llsa_b200
    q, k, v, do = _operands(layout)
    table, w = torch.ones(2048, 64, device=DEV, dtype=q.dtype), torch.ones(64, device=DEV, requires_grad=True)
    for front, two in (((None, None, None, 0.0), 0), ((None, None, None, 0.0), 8), ((table, w, w, 1e-5), 0)):
        torch.library.opcheck(L.layer_fwd.default, (q, k, v, *front, 8, two, 16, 2 if two else 1),
                              test_utils=("test_schema", "test_faketensor", "test_autograd_registration", "test_aot_dispatch_static"))
    q, k, v, w = [t.detach() for t in (q, k, v, w)]
    which = ("test_schema", "test_faketensor")
    o, saved, qr, kr = L.layer_fwd(q, k, v, table, w, w, 1e-5, 8, 0, 16, 1)
    torch.library.opcheck(L.layer_bwd.default, (do, qr, kr, v, o, saved, table, q, k, w, w, 1e-5, 8, 0, 16, 1, True), test_utils=which)
    one, two = llsa_b200.llsa_l1_debug(q, k, v, 8, 16), llsa_b200.llsa_l2_debug(q, k, v, 8, 8, 16)
    for dbg, low, lists in ((one, (None, None), (None, 8, 0)), (two, (two["pk2"], two["pv2"]), (two["p_indices"], 8, 8))):
        args = (q, k, v, dbg["pk"], dbg["pv"], *low)
        torch.library.opcheck(L.attn_fwd.default, args + (dbg["indices"], *lists, 16, 16.0, 256.0), test_utils=which)
        torch.library.opcheck(L.attn_bwd.default, (do, *args, dbg["o"], dbg["lse"], dbg["indices"], *lists, 16, 16.0, 256.0, 16.0, 256.0, False),
                              test_utils=which)
